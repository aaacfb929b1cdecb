// The FP64 collision of one cell in block fixed point: 64-bit integers over one
// exponent per cell.
//
// GB300 has two FP64 lanes per SM (measured 2.0 DFMA, 1.7 DADD and also 2.0
// double <-> int64 conversions per clock and SM), against 64 integer additions
// and about 18 32 x 32 -> 64-bit multiply-adds.  A D3Q27 update in FP64
// arithmetic takes 133 instructions of that pipe; here it takes the 54
// conversions (27 in, 27 out) and everything between runs on the integer pipes.
//
// Format.  The weights of both lattices are one constant W times powers of two
// (D3Q27: 1/27 x {8, 2, 1/2, 1/8}; D2Q9: 1/9 x {4, 1, 1/4}), so g_i = f_i 2^-k_i
// removes them from the equilibrium: with om = omega,
//   g_i' = (1 - om) g_i + [G + sum_a e_a^2 Q_aa + 2 sum_{a<b} e_a e_b Q_ab]
//                       + [e . V],
//   Q_ab = 4.5 W om u_a u_b,  V_a = 3 W om u_a,  G = W om rho3 - (sum_a Q_aa) / 3,
// the relaxation toward w_i (rho3 + 3 e.u + 4.5 (e.u)^2 - 1.5 u^2), additions
// only from here on except one product per population.  E is the exponent of the
// largest |g_i| of the cell; q_i = g_i 2^(55 - E), rounded to nearest: 55
// significant bits at the largest population.  The moments are exact integer
// sums of the q_i (headroom: 216 x 2^56 < 2^64 in units of the corner weight, rho3
// at half that scale), the products are rounded 64 x 64 -> 64-bit high parts
// with constants of 58 to 63 bits, and the relaxed populations come out in units
// of 2^(E - 54), which one conversion rounds to 53 bits.  Every rounding is to
// nearest, so no step adds a bias.
//
// Cells the format does not cover take the FP64 operations (bgk_relax_each):
// |g_i| >= 1/4 (|u| well above 0.3), infinities and NaNs, and rates within 2^-20
// of 0 or 2.  Below 2^-900 the exponent stays at -900.
#pragma once
#include "solver.cuh"

namespace cflbm {

constexpr int FX_P = 55;             // q_i = g_i 2^(FX_P - E)
constexpr int FX_EMAX = 1023 - 3;    // largest biased exponent covered
constexpr int FX_EMIN = 1023 - 900;  // smaller ones are raised to it
// Populations 0 .. FX_NINT - 1 are converted to FP64 with integer operations, the
// others by the FP64 pipe: with all 54 conversions of a D3Q27 cell on it that pipe
// binds (27 clocks per cell and SM), with all 27 outgoing ones off it the integer
// pipes do.  10 steps and the fields of the 512x128x128 cylinder, ms: 9.34 / 8.86
// / 8.54 / 8.46 / 8.39 / 8.48 / 8.70 for 0 / 6 / 10 / 14 / 18 / 22 / 27 (FP64
// operations: 22.78); REF3D 257x97x97, 20 steps: 6.43 / 6.02 / 5.80 / 5.65 / 5.51
// / 5.43 / 5.58 (15.17); D2Q9 400x100, 400 steps: 2.78 ms for none, 2.70 for all 9
// (3.11).
template <class L> constexpr int fx_nint = L::D == 3 ? 18 : 4;

// Shift of the weight of class c = |e|^2 (w = W 2^k), the scale of the velocity
// sums (u = M 2^(E - FX_P - FX_U)) and of rho3 (FX_R).
template <class L> struct Fx {
  static constexpr int k(int c) { return (L::D == 3 ? 3 : 2) - 2 * c; }
  static constexpr int U = L::D == 3 ? 3 : 4;
  static constexpr int R = 2;
};

// 64-bit integer as balanced limbs h 2^32 + l, both signed.
struct Limbs {
  int h, l;
};
__device__ __forceinline__ Limbs limbs(long long x) {
  const unsigned lo = (unsigned)x;
  return {(int)(x >> 32) + (int)(lo >> 31), (int)lo};
}
// x c / 2^64 + add, rounded to nearest but for the product of the low limbs
// (below a quarter of a unit, of either sign).
__device__ __forceinline__ long long mul_hi(Limbs x, FxConst c, long long add) {
  long long cross = (long long)x.l * c.h + 0x80000000LL;
  cross = (long long)x.h * c.l + cross;
  return (long long)x.h * c.h + ((cross >> 32) + add);
}
__device__ __forceinline__ long long mul_hi(long long x, FxConst c, long long add = 0) {
  return mul_hi(limbs(x), c, add);
}
__device__ __forceinline__ long long mul_hi(Limbs x, Limbs y, long long add) {
  return mul_hi(x, FxConst{y.h, y.l}, add);
}

// Larger magnitude of two doubles' high words, as floats: the order of
// magnitudes is the words' order, and a word that is a float NaN (|d| >= 2^1017,
// infinities and NaNs among them) wins.
__device__ __forceinline__ float max_mag(float m, double d) {
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(m), "f"(fabsf(__int_as_float(__double2hiint(d)))));
  return r;
}

// Biased exponent of the cell's largest |g_i| (at least FX_EMIN); `ux` takes part
// as a velocity that replaces the cell's (0: none).
template <class L>
__device__ __forceinline__ int fx_exponent(const double *f, double ux) {
  float m[L::D + 1] = {};
  static_for(
      [&](auto ic) {
        constexpr int I = decltype(ic)::value;
        m[wclass<L>(I)] = max_mag(m[wclass<L>(I)], f[I]);
      },
      std::make_integer_sequence<int, L::Q>{});
  // |ux| <= 8 max |g| keeps its integer below 2^62
  int hi = (__double2hiint(ux) & 0x7FFFFFFF) - (3 << 20);
#pragma unroll
  for (int c = 0; c <= L::D; ++c) hi = max(hi, __float_as_int(m[c]) - Fx<L>::k(c) * (1 << 20));
  return max(hi >> 20, FX_EMIN);
}

// d 2^s by its exponent field (d zero or far below 1 when the result is).
__device__ __forceinline__ double scale_bits(double d, int s20) {
  return __hiloint2double(__double2hiint(d) + s20, __double2loint(d));
}

// x 2^(s20 / 2^20 - 1023) in FP64 (s20: the biased exponent of 1 in x's units, at
// bit 20), rounded to nearest, on the integer pipes: 17 operations for the
// conversion's slot of the FP64 pipe.
__device__ __forceinline__ double fx_to_double(long long x, int s20) {
  const long long sg = x >> 63;
  unsigned long long u = (unsigned long long)((x ^ sg) - sg);
  const int z = __clzll((long long)u);
  u = z < 64 ? u << z : 0;
  const unsigned long long m = (u >> 11) + ((u >> 10) & 1);
  const unsigned long long r = m + ((unsigned long long)(unsigned)(s20 + ((62 - z) << 20)) << 32);
  return __longlong_as_double(u == 0 ? 0 : (long long)(r | ((unsigned long long)sg << 63)));
}

// The populations as integers q_i and their moments: the cascade of moments_get
// with the weights' factor 4 between a line's middle and its ends.
template <class L>
__device__ __forceinline__ void fx_moments(const double *f, int eb, long long *q, long long &mr,
                                           long long *mu) {
  const int in20 = (FX_P + 1023 - eb) << 20;
  static_for(
      [&](auto ic) {
        constexpr int I = decltype(ic)::value;
        q[I] = __double2ll_rn(scale_bits(f[I], in20 - Fx<L>::k(wclass<L>(I)) * (1 << 20)));
      },
      std::make_integer_sequence<int, L::Q>{});
  if constexpr (L::D == 3) {
    long long s0[3][3], s1[3][3];
    static_for(
        [&](auto kc) {
          constexpr int k = decltype(kc)::value, i = k / 3, j = k % 3;
          const long long lo = q[dir_of<L>(i - 1, j - 1, -1)], hi = q[dir_of<L>(i - 1, j - 1, 1)];
          s0[i][j] = lo + hi + 4 * q[dir_of<L>(i - 1, j - 1, 0)];
          s1[i][j] = hi - lo;
        },
        std::make_integer_sequence<int, 9>{});
    long long t00[3], t01[3], t10[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      t00[i] = s0[i][0] + s0[i][2] + 4 * s0[i][1];
      t01[i] = s0[i][2] - s0[i][0];
      t10[i] = s1[i][0] + s1[i][2] + 4 * s1[i][1];
    }
    mr = ((t00[0] + t00[2]) >> 1) + 2 * t00[1];
    mu[0] = t00[2] - t00[0];
    mu[1] = t01[0] + t01[2] + 4 * t01[1];
    mu[2] = t10[0] + t10[2] + 4 * t10[1];
  } else {
    long long s0[3], s1[3];
    static_for(
        [&](auto kc) {
          constexpr int i = decltype(kc)::value;
          const long long lo = q[dir_of<L>(i - 1, -1, 0)], hi = q[dir_of<L>(i - 1, 1, 0)];
          s0[i] = lo + hi + 4 * q[dir_of<L>(i - 1, 0, 0)];
          s1[i] = hi - lo;
        },
        std::make_integer_sequence<int, 3>{});
    mr = s0[0] + s0[2] + 4 * s0[1];
    mu[0] = 4 * (s0[2] - s0[0]);
    mu[1] = 4 * (s1[0] + s1[2] + 4 * s1[1]);
    mu[2] = 0;
  }
}

// u, v, w and p = rho3 / 3 of one cell in FP64 (null pointers: not wanted).
template <class L>
__device__ __forceinline__ void fx_store_macros(const SweepArgs &a, long long cell, int eb,
                                                long long mr, const long long *mu) {
  const double su = __hiloint2double((eb - FX_P - Fx<L>::U) << 20, 0);
  const double sr = __hiloint2double((eb - FX_P - Fx<L>::R) << 20, 0);
  if (a.mu) a.mu[cell] = __dmul_rn(__ll2double_rn(mu[0]), su);
  if (a.mv) a.mv[cell] = __dmul_rn(__ll2double_rn(mu[1]), su);
  if (a.mw) a.mw[cell] = __dmul_rn(__ll2double_rn(mu[2]), su);
  if (a.mp) a.mp[cell] = __ddiv_rn(__dmul_rn(__ll2double_rn(mr), sr), 3.0);
}

// Collision and store of one cell with FP64 arithmetic.  f: the pulled
// populations.  solid: p = u = 0; inlet: u = (ux_in, 0, 0); outlet: p = 0 (the
// reference profiles' rules).  Returns false, with nothing written, where the
// format does not cover the cell.
template <class L, class SF, class E>
__device__ __forceinline__ bool fixed_cell(const double *f, bool solid, bool inlet, double ux_in,
                                           bool outlet, long long cell, bool store,
                                           E *__restrict__ fb, long long c, long long S,
                                           const SweepArgs &a) {
  constexpr int D = L::D;
  const int eb = fx_exponent<L>(f, inlet && !solid ? ux_in : 0.0);
  double s = 1.0;
  if (a.alpha) s = __dsub_rn(1.0, (double)a.alpha[cell]);
  if (!a.fx_ok || eb > FX_EMAX || !(fabs(s) <= 1.0)) return false;

  long long q[L::Q], mr, mu[3];
  fx_moments<L>(f, eb, q, mr, mu);
  if (solid) mr = mu[0] = mu[1] = mu[2] = 0;
  if (inlet) {
    mu[0] = __double2ll_rn(scale_bits(ux_in, (FX_P + Fx<L>::U + 1023 - eb) << 20));
    mu[1] = mu[2] = 0;
  }
  if (outlet) mr = 0;

  if (a.mu && store) fx_store_macros<L>(a, cell, eb, mr, mu);
  if (a.alpha) {  // u (1 - alpha): the factor at 2^62, the product back by 4
    const Limbs sl = limbs(__double2ll_rn(__dmul_rn(s, 4611686018427387904.0)));
#pragma unroll
    for (int d = 0; d < D; ++d) mu[d] = 4 * mul_hi(limbs(mu[d]), sl, 0);
  }

  // Q_ab and V_a in units of 2^(E - 54).
  const int n = min(2 * Fx<L>::U - 9 + 1023 - eb, 63);
  const long long half = (1LL << n) >> 1;
  long long qd[D], qo[D == 3 ? 3 : 1], v[D];
  {
    Limbs ml[D], tl[D];
#pragma unroll
    for (int d = 0; d < D; ++d) {
      ml[d] = limbs(mu[d]);
      tl[d] = limbs(mul_hi(ml[d], a.fx[FX_T], 0));
      v[d] = mul_hi(ml[d], a.fx[FX_V], 0);
    }
#pragma unroll
    for (int d = 0; d < D; ++d) qd[d] = mul_hi(tl[d], ml[d], half) >> n;
    qo[0] = 2 * (mul_hi(tl[0], ml[1], half) >> n);  // 2 Q_xy
    if constexpr (D == 3) {
      qo[1] = 2 * (mul_hi(tl[0], ml[2], half) >> n);  // 2 Q_xz
      qo[2] = 2 * (mul_hi(tl[1], ml[2], half) >> n);  // 2 Q_yz
    }
  }
  long long qs = qd[0] + qd[1];
  if constexpr (D == 3) qs += qd[2];
  const long long G = mul_hi(mr, a.fx[FX_G], -mul_hi(qs, a.fx[FX_THIRD]));

  const int out20 = (eb - 1023 - (FX_P - 1)) * (1 << 20);
  auto put = [&](auto ic, long long eq) {
    constexpr int I = decltype(ic)::value;
    const long long x = mul_hi(q[I], a.fx[FX_OMC], eq);
    double r;
    if constexpr (I < fx_nint<L>) {
      r = fx_to_double(x, out20 + (1023 + Fx<L>::k(wclass<L>(I))) * (1 << 20));
    } else {
      const double d = __ll2double_rn(x);
      const int hi = __double2hiint(d);
      r = __hiloint2double(hi == 0 ? 0 : hi + (out20 + Fx<L>::k(wclass<L>(I)) * (1 << 20)),
                           __double2loint(d));
    }
    if (store)
      SF::template store<double, L>(fb + I * S + c, r, a.L.fbase[I], (unsigned)(cell * L::Q + I),
                                    a.f16_sr);
  };
  put(std::integral_constant<int, 0>{}, G);
  static_for(
      [&](auto kc) {
        constexpr int k = decltype(kc)::value;
        constexpr int i = L::pair(k), j = L::opp(L::pair(k));
        constexpr int ex = L::ex(i), ey = L::ey(i), ez = L::ez(i);
        long long even = G, odd = 0;
        if constexpr (ex != 0) {
          even += qd[0];
          odd = ex > 0 ? v[0] : -v[0];
        }
        if constexpr (ey != 0) {
          even += qd[1];
          odd = ey > 0 ? odd + v[1] : odd - v[1];
        }
        if constexpr (D == 3 && ez != 0) {
          even += qd[D - 1];
          odd = ez > 0 ? odd + v[D - 1] : odd - v[D - 1];
        }
        if constexpr (ex * ey != 0) even = ex * ey > 0 ? even + qo[0] : even - qo[0];
        if constexpr (D == 3) {
          if constexpr (ex * ez != 0) even = ex * ez > 0 ? even + qo[1] : even - qo[1];
          if constexpr (ey * ez != 0) even = ey * ez > 0 ? even + qo[2] : even - qo[2];
        }
        put(std::integral_constant<int, i>{}, even + odd);
        put(std::integral_constant<int, j>{}, even - odd);
      },
      std::make_integer_sequence<int, L::NPAIR>{});
  return true;
}

}  // namespace cflbm

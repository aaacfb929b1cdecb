// The FP64 collision of one cell in block fixed point: 64-bit integers over one
// exponent per cell.
//
// GB300 has two FP64 lanes per SM (measured 2.0 DFMA, 1.7 DADD and also 2.0
// double <-> int64 conversions per clock and SM), against 64 integer additions
// and about 18 32 x 32 -> 64-bit multiply-adds.  A D3Q27 update in FP64
// arithmetic takes 133 instructions of that pipe; here it takes 32 conversions (27
// in, 5 out; fx_pipe) and everything else runs on the integer pipes.
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
// of 2^(E - 54), which one conversion rounds to 53 bits.  Roundings are to nearest,
// ties up in the products, to even in the FP64 pipe's conversions and away from zero in
// the integer one (at the largest populations two bits are dropped, so a quarter of
// those values are ties); rho3's half is floored.
//
// Cells the format does not cover take the FP64 operations (bgk_relax_each):
// |g_i| >= 1/4 (|u| well above 0.3), infinities and NaNs, and rates within 2^-20
// of 2 or, with FP64 (not DF64) arithmetic, below 1.1 (D3Q27) or 0.69 (D2Q9) (see
// set_relax).  Below 2^-900 the exponent stays at -900.
#pragma once
#include "solver.cuh"

namespace cflbm {

constexpr int FX_P = 55;             // q_i = g_i 2^(FX_P - E)
constexpr int FX_EMAX = 1023 - 3;    // largest biased exponent covered
constexpr int FX_EMIN = 1023 - 900;  // smaller ones are raised to it
// Populations that the FP64 pipe converts back; the others are converted with integer
// operations: with all 54 conversions of a D3Q27 cell on that pipe it binds (27 clocks
// per cell and SM), with all 27 outgoing ones off it the integer pipes do.  10 steps and
// the fields of the 512x128x128 cylinder, ms: 7.50 / 7.40 / 7.33 / 7.36 / 7.39 with 9 / 7
// / 5 / 2 / 0 there (with a longer conversion 9.34 for 27, 8.39 for 9; FP64 operations:
// 22.78); D2Q9 1132x168, 400 steps: 3.31 / 3.24 / 3.22 / 3.25 with 6 / 5 / 4 / 3 (FP64
// operations: 4.01).  The two round ties differently (to even; away from zero), so the
// set holds with a direction its mirror images: populations that are equal stay equal,
// and a flow uniform in z keeps w = 0.  Of such sets in D3Q27, rest and the yz / xz / xy
// diagonals, rest and the x and y axes: 649 / 659 / 660 / 668 us per step at 512x128x128
// (the last five by index, not closed: 666), 19.3 / 19.6 / 20.4 / 20.3 at 100x40x36
// (19.9), REF3D 257x97x97 223.5 / 223.8 / 227.2 / 226.6 (226.3).
template <class L>
__host__ __device__ constexpr bool fx_pipe(int i) {
  return L::D == 3 ? i == 0 || (L::ex(i) == 0 && wclass<L>(i) == 2) : wclass<L>(i) == 2;
}

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
// x c / 2^64 + add + 2^31, rounded to nearest but for the product of the low limbs
// (below a quarter of a unit, of either sign).  The cross terms carry 2^63 so that
// their upper word needs no sign extension; callers take the FX_BIAS off once.
constexpr long long FX_BIAS = 1LL << 31;
__device__ __forceinline__ long long mul_hi_b(Limbs x, FxConst c, long long add) {
  unsigned long long cross = (unsigned long long)((long long)x.l * c.h) + 0x8000000080000000ULL;
  cross += (unsigned long long)((long long)x.h * c.l);
  return (long long)x.h * c.h + (add + (long long)(cross >> 32));
}
__device__ __forceinline__ long long mul_hi(Limbs x, FxConst c, long long add) {
  return mul_hi_b(x, c, add - FX_BIAS);
}
__device__ __forceinline__ long long mul_hi(long long x, FxConst c, long long add = 0) {
  return mul_hi(limbs(x), c, add);
}
__device__ __forceinline__ long long mul_hi(Limbs x, Limbs y, long long add) {
  return mul_hi(x, FxConst{y.h, y.l}, add);
}

// Larger of m and the magnitudes of two doubles' high words, as floats: the order of
// magnitudes is the words' order, and a word that is a float NaN (|d| >= 2^1017,
// infinities and NaNs among them) wins.
__device__ __forceinline__ float max_mag(float m, double d, double e) {
  float r;
  asm("max.NaN.f32 %0, %1, %2, %3;"
      : "=f"(r)
      : "f"(m), "f"(fabsf(__int_as_float(__double2hiint(d)))),
        "f"(fabsf(__int_as_float(__double2hiint(e)))));
  return r;
}

// Biased exponent of the cell's largest |g_i| (at least FX_EMIN); `ux` takes part
// as a velocity that replaces the cell's (0: none).
template <class L>
__device__ __forceinline__ int fx_exponent(const double *f, double ux) {
  float m[L::D + 1] = {};
  static_for(
      [&](auto kc) {
        constexpr int i = L::pair(decltype(kc)::value), c = wclass<L>(i);
        m[c] = max_mag(m[c], f[i], f[L::opp(i)]);
      },
      std::make_integer_sequence<int, L::NPAIR>{});
  m[0] = max_mag(0.0f, f[0], f[0]);
  // ux's integer, 2^(FX_P + U - E) ux, stays below 2^62
  int hi = (__double2hiint(ux) & 0x7FFFFFFF) - ((6 - Fx<L>::U) << 20);
#pragma unroll
  for (int c = 0; c <= L::D; ++c) {
    int h = __float_as_int(m[c]);
    if (Fx<L>::k(c) < 0) h = min(h, 0x7F800000);  // NaNs as infinity: below 2^31 shifted
    hi = max(hi, h - Fx<L>::k(c) * (1 << 20));
  }
  return max(hi >> 20, FX_EMIN);
}

// d 2^s by its exponent field (d zero or far below 1 when the result is).
__device__ __forceinline__ double scale_bits(double d, int s20) {
  return __hiloint2double(__double2hiint(d) + s20, __double2loint(d));
}

// x 2^(s20 / 2^20 - 1023) in FP64 (s20: the biased exponent of 1 in x's units, at
// bit 20; |x| < 2^63), rounded to nearest, on the integer pipes.
__device__ __forceinline__ double fx_to_double(long long x, int s20) {
  unsigned lo = (unsigned)x;
  const unsigned sign = (unsigned)(x >> 32);
  unsigned hi = sign;
  asm("{\n\t.reg .pred p;\n\t"
      "setp.lt.s32 p, %1, 0;\n\t"
      "@p sub.cc.u32 %0, 0, %0;\n\t"
      "@p subc.u32 %1, 0, %1;\n\t}"
      : "+r"(lo), "+r"(hi));
  const bool low = hi == 0u;
  const int z = __clz((int)(low ? lo : hi)) + (low ? 31 : -1);  // to bit 62; 63 for zero
  unsigned long long u = (((unsigned long long)hi << 32) | lo) << z;
  u = (u + 0x200u) >> 10;  // 53 bits, the first one included; a carry enters the exponent
  const int e = z == 63 ? 0 : s20 + ((61 - z) << 20);
  return __hiloint2double((int)(((unsigned)(u >> 32) + (unsigned)e) | (sign & 0x80000000u)),
                          (int)(unsigned)u);
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

// u, v, w and p = rho3 / 3 of one cell in FP64 (null pointers: not wanted), without
// the FP64 pipe: its conversions, scalings and the division took half its time in
// macros_channel_kernel (512x128x128: 640 -> 420 us).
template <class L>
__device__ __forceinline__ void fx_store_macros(const SweepArgs &a, long long cell, int eb,
                                                long long mr, const long long *mu) {
  const int su = (eb - FX_P - Fx<L>::U) * (1 << 20), sr = (eb - FX_P - Fx<L>::R) * (1 << 20);
  if (a.mu) a.mu[cell] = fx_to_double(mu[0], su);
  if (a.mv) a.mv[cell] = fx_to_double(mu[1], su);
  if (a.mw) a.mw[cell] = fx_to_double(mu[2], su);
  if (a.mp) a.mp[cell] = fx_to_double(mul_hi(mr, a.fx[FX_THIRD]), sr);
}

// Collision and store of one cell with FP64 arithmetic, population i to
// fb[doff_i + at] (fb: the block's first cell).  f: the pulled populations.  solid: p = u = 0; inlet: u = (ux_in, 0, 0); outlet: p = 0 (the
// reference profiles' rules).  MACROS: fields out, where the step wants them.
// Returns false, with nothing written, where the
// format does not cover the cell.
template <class L, class SF, bool MACROS, class E>
__device__ __forceinline__ bool fixed_cell(const double *f, bool solid, bool inlet, double ux_in,
                                           bool outlet, long long cell, bool store,
                                           E *__restrict__ fb, unsigned at,
                                           const SweepArgs &a) {
  constexpr int D = L::D;
  const int eb = fx_exponent<L>(f, inlet ? ux_in : 0.0);
  double s = 1.0;
  if (a.alpha && store) s = __dsub_rn(1.0, (double)a.alpha[cell]);
  // (lanes that store nothing hold padding, which may be anything: never a reason)
  if (!a.fx_ok || eb > FX_EMAX || !(fabs(s) <= 1.0)) return !store && a.fx_ok;

  long long q[L::Q], mr, mu[3];
  fx_moments<L>(f, eb, q, mr, mu);
  if (solid) mr = mu[0] = mu[1] = mu[2] = 0;
  if (inlet) {
    mu[0] = __double2ll_rn(scale_bits(ux_in, (FX_P + Fx<L>::U + 1023 - eb) << 20));
    mu[1] = mu[2] = 0;
  }
  if (outlet) mr = 0;

  if constexpr (MACROS)
    if (a.mu && store) fx_store_macros<L>(a, cell, eb, mr, mu);
  if (a.alpha) {  // u (1 - alpha): the factor at 2^62, the product back by 4
    const Limbs sl = limbs(__double2ll_rn(__dmul_rn(s, 4611686018427387904.0)));
#pragma unroll
    for (int d = 0; d < D; ++d) mu[d] = 4 * mul_hi(limbs(mu[d]), sl, 0);
  }

  // Q_ab and V_a in units of 2^(E - 54).
  const int n = min(2 * Fx<L>::U - 9 + 1023 - eb, 63);
  const long long half = (long long)((1ULL << n) >> 1);
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
  // less the bias that every population's product adds (mul_hi_b)
  const long long G = mul_hi(mr, a.fx[FX_G], -mul_hi(qs, a.fx[FX_THIRD])) - FX_BIAS;

  const int out20 = (eb - 1023 - (FX_P - 1)) * (1 << 20);
  auto put = [&](auto ic, long long eq) {
    constexpr int I = decltype(ic)::value;
    const long long x = mul_hi_b(limbs(q[I]), a.fx[FX_OMC], eq);
    double r;
    if constexpr (!fx_pipe<L>(I)) {
      r = fx_to_double(x, out20 + (1023 + Fx<L>::k(wclass<L>(I))) * (1 << 20));
    } else {
      const double d = __ll2double_rn(x);
      const int hi = __double2hiint(d);
      r = __hiloint2double(hi == 0 ? 0 : hi + (out20 + Fx<L>::k(wclass<L>(I)) * (1 << 20)),
                           __double2loint(d));
    }
    if (store)
      SF::template store<double, L>(fb + a.doff[I] + at, r, a.L.fbase[I],
                                    (unsigned)(cell * L::Q + I), a.f16_sr);
  };
  auto pair = [&](auto kc, long long even, long long odd) {  // direction i and its opposite
    constexpr int i = L::pair(decltype(kc)::value);
    put(std::integral_constant<int, i>{}, even + odd);
    put(std::integral_constant<int, L::opp(i)>{}, even - odd);
  };
  // pair index of velocity (x, y, z) or of its opposite; the odd part's sign
  auto dir = [&](auto xc, auto yc, auto zc, long long even, long long odd) {
    constexpr int i = dir_of<L>(decltype(xc)::value, decltype(yc)::value, decltype(zc)::value);
    constexpr int k = pair_of<L>(i);
    pair(std::integral_constant<int, k>{}, even, L::pair(k) == i ? odd : -odd);
  };
  using P1 = std::integral_constant<int, 1>;
  using N1 = std::integral_constant<int, -1>;
  using Z0 = std::integral_constant<int, 0>;
  put(std::integral_constant<int, 0>{}, G);
  const long long ex = G + qd[0], ey = G + qd[1], exy = ex + qd[1];
  const long long vp = v[0] + v[1], vm = v[0] - v[1];
  dir(P1{}, Z0{}, Z0{}, ex, v[0]);
  dir(Z0{}, P1{}, Z0{}, ey, v[1]);
  dir(P1{}, P1{}, Z0{}, exy + qo[0], vp);
  dir(P1{}, N1{}, Z0{}, exy - qo[0], vm);
  if constexpr (D == 3) {
    const long long exz = ex + qd[2], eyz = ey + qd[2], e3 = exy + qd[2];
    const long long sp = qo[1] + qo[2], sm = qo[1] - qo[2];  // 2 (Q_xz +- Q_yz)
    dir(Z0{}, Z0{}, P1{}, G + qd[2], v[2]);
    dir(P1{}, Z0{}, P1{}, exz + qo[1], v[0] + v[2]);
    dir(P1{}, Z0{}, N1{}, exz - qo[1], v[0] - v[2]);
    dir(Z0{}, P1{}, P1{}, eyz + qo[2], v[1] + v[2]);
    dir(Z0{}, P1{}, N1{}, eyz - qo[2], v[1] - v[2]);
    const long long ep = e3 + qo[0], em = e3 - qo[0];
    dir(P1{}, P1{}, P1{}, ep + sp, vp + v[2]);
    dir(P1{}, P1{}, N1{}, ep - sp, vp - v[2]);
    dir(P1{}, N1{}, P1{}, em + sm, vm + v[2]);
    dir(P1{}, N1{}, N1{}, em - sm, vm - v[2]);
  }
  return true;
}

}  // namespace cflbm

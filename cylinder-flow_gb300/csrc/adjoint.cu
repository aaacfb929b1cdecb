// Discrete adjoint of the D2Q9 channel step (the differentiation form).
//
// Objective: J = mean over steps t0..t1 of the body force F_x (or F_y), where
// step t's force is the momentum exchange of state s_t, the post-collision
// field the t-th sweep reads.  Parameters: the per-cell Brinkman porosity
// alpha, the inlet speed u_in (inlet equilibrium and initial velocity) and the
// relaxation time tau = tau0 + 0.5 (omega = 1/tau).
//
// Forward: s_1 = C(feq(U0)), and s_{t+1} = C(g_{t+1}) with g_{t+1} = P s_t, P
// the boundary-resolving pull (plain shift, inlet equilibrium, zero-gradient
// outlet, free-slip mirror / no-slip / periodic y walls, halfway bounce-back on
// solids) and C the cellwise BGK collision toward feq(rho, (1 - alpha) u).
// With lambda_t = dJ/ds_t and mu^{t+1} = C'(g_{t+1})^T lambda_{t+1}:
//   lambda_t = P^T mu^{t+1} + c_t dF_t/ds_t       (c_t = 1/(t1-t0+1) in the window)
// The reverse sweep for state s_t is one fused kernel per cell X: gather
// lambda_{t+1}(X) from mu^{t+2} (a plain shift for regular cells; cells on the
// box faces or next to the body enumerate every neighbour (Y, i) whose pull
// source is X, i.e. bounce-back reverses into X's own opposite population),
// recompute g_{t+1}(X) = (P s_t)(X), and write mu^{t+1}(X) with the
// sensitivities of C and of the inlet pulls.  States come from checkpoints
// every K steps, recomputed one segment at a time into two alternating segment
// buffers: memory ceil(T/K) + 2K states.
// Sensitivity sums are deterministic: alpha per cell (arithmetic type within a
// segment, FP64 across segments), omega and u_in per block in FP64.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>
#include "float_limbs.hpp"
#include "handle.hpp"

namespace cflbm {
int record_error(int code, const char *msg);
}
using namespace cflbm;

namespace {

// D2Q9 velocities (0; +x, +y, -x, -y; diagonals 5..8), opposites and y mirrors
// as functions, usable with run-time indices in device code.
__host__ __device__ constexpr int AXf(int i) {
  return (i == 1 || i == 5 || i == 8) ? 1 : ((i == 3 || i == 6 || i == 7) ? -1 : 0);
}
__host__ __device__ constexpr int AYf(int i) {
  return (i == 2 || i == 5 || i == 6) ? 1 : ((i == 4 || i == 7 || i == 8) ? -1 : 0);
}
__host__ __device__ constexpr int AOPPf(int i) {
  return i == 0 ? 0 : (i < 5 ? (i + 1) % 4 + 1 : (i - 3) % 4 + 5);
}
__host__ __device__ constexpr int AMYf(int i) {
  return i == 2 ? 4 : i == 4 ? 2 : i == 5 ? 8 : i == 8 ? 5 : i == 6 ? 7 : i == 7 ? 6 : i;
}
__host__ __device__ constexpr double aw(int i) {
  return i == 0 ? 4.0 / 9.0 : (i < 5 ? 1.0 / 9.0 : 1.0 / 36.0);
}

constexpr int ABX = 32, ABY = 4, ANT = ABX * ABY;

// Interior segments from which their units are captured and replayed: a capture
// and its instantiation cost about what launching a unit 4 times directly does.
constexpr int GRAPH_UNITS = 8;

constexpr int GMAX = 4;  // contributions per (cell, population) in the adjoint gather

struct AdjArgs {
  Layout L;                        // state layout
  const void *s;                   // s_t
  const void *mu_next;             // mu^{t+2}, dense [i][y][x]
  void *mu_out;                    // mu^{t+1}, dense (final gather: lambda_1)
  const uint32_t *mask;            // solid mask (bit-packed)
  int nxw;
  const int *aux;                  // per cell: AUX_SOLID, AUX_REGULAR or irregular entry r
  // Per entry, population j's byte (cell_code) at byte j % 4 of word j / 4,
  // words [..][3][entry]: GMAX contributions to lambda (CODE_NONE: none), and the
  // pull source (CODE_INLET + p: inlet population p).
  const unsigned *gat;
  const unsigned *pul;
  int nirr;                        // entries
  const unsigned *lkr;             // per entry: link bits (bit i: source of i is solid), and
                                   // bit 31 when a population has more than one contribution
  const float *alpha;              // Brinkman porosity or null
  double omega;
  double u_in;
  // Inlet populations and their derivatives by u_in, formed on the host: in the
  // kernel their FP64 operations, for one lane of the first column's warps, took
  // 3 us of the launch (the SMs holding those blocks had their FP64 pipe 98 % busy).
  double fin[9], dfin[9];
  float fin_f[9];
  double c_next;                   // objective weight of step t+1 (when seg is null)
  const int *seg;                  // device: index k of the segment being reversed
  const double *c_tab;             // objective weight of every step 0..T+1
  int K;                           // checkpoint spacing
  int q;                           // state s_t of this launch: t = k*K + 1 + q
  int obj_axis;                    // 0: F_x, 1: F_y
  void *g_alpha;                   // per cell, arithmetic type (segment accumulator)
  double *g_block;                 // per block: [0] omega, [1] u_in (FP64, owned)
};

// A population p of a cell one step (dx, dy) away (periodic rows wrap), in a byte.
enum { CODE_INLET = 0xF0, CODE_NONE = 0xFF };
__device__ __forceinline__ unsigned cell_code(int p, int dx, int dy) {
  return (unsigned)(p << 4 | (dy + 1) << 2 | (dx + 1));
}

enum { SRC_CELL = 0, SRC_INLET = 1 };
enum { AUX_SOLID = -2, AUX_REGULAR = -1 };

// Link bits of cell (x, y): bit i set when the pull of population i meets a solid.
__device__ __forceinline__ unsigned link_bits(const uint32_t *mask, int nxw, int nx, int ny,
                                              int wall_y, int x, int y) {
  unsigned b = 0;
  for (int i = 1; i < 9; ++i) {
    int sx = x - AXf(i), sy = y - AYf(i);
    if (sy < 0 || sy >= ny) {
      if (wall_y == WALL_PERIODIC) sy = sy < 0 ? sy + ny : sy - ny;
      else if (wall_y == WALL_FREESLIP) sy = y;
      else continue;
    }
    if (sx < 0) continue;
    if (sx >= nx) sx = nx - 1;
    if (mask_solid(mask, nxw, ny, sx, sy, 0)) b |= 1u << i;
  }
  return b;
}

// Pull source of population i at fluid cell (x, y): the forward channel pull
// for D2Q9 (sweep.cuh, pull_resolved) with the configured y walls.  SRC_CELL:
// population j of (sx, sy) (bounce-back: the cell's own opposite population).
// SRC_INLET: inlet equilibrium population j.  lk: the cell's link bits.
__device__ __forceinline__ int pull_source(int nx, int ny, int wall_y, unsigned lk, int x, int y,
                                           int i, int &sx, int &sy, int &j) {
  if (i == 0) {
    sx = x; sy = y; j = 0;
    return SRC_CELL;
  }
  sx = x - AXf(i);
  sy = y - AYf(i);
  j = i;
  bool bb = false;
  if (sy < 0 || sy >= ny) {
    if (wall_y == WALL_PERIODIC) sy = sy < 0 ? sy + ny : sy - ny;
    else if (wall_y == WALL_FREESLIP) { j = AMYf(i); sy = y; }
    else bb = true;
  }
  if (bb || ((lk >> i) & 1u)) {
    sx = x; sy = y; j = AOPPf(i);
    return SRC_CELL;
  }
  if (sx < 0) return SRC_INLET;
  if (sx >= nx) sx = nx - 1;
  return SRC_CELL;
}

inline double inlet_f(int j, double u) {
  const double e = AXf(j) * u;
  return aw(j) * (3.0 * e + 4.5 * e * e - 1.5 * u * u);
}
inline double inlet_dfdu(int j, double u) {
  return aw(j) * (3.0 * AXf(j) + 9.0 * AXf(j) * AXf(j) * u - 3.0 * u);
}

// Block sum of an FP64 value; valid in thread 0 of the block.
__device__ __forceinline__ double block_sum(double v, double *sh) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  const int tid = threadIdx.y * ABX + threadIdx.x;
  __syncthreads();
  if ((tid & 31) == 0) sh[tid >> 5] = v;
  __syncthreads();
  double s = 0.0;
  if (tid == 0)
    for (int w = 0; w < ANT / 32; ++w) s += sh[w];
  return s;
}

// Block sum of an FP32 value, at least as accurate as FP64 additions, without the FP64
// pipe (two lanes per SM: the shuffle tree of FP64 additions took 4 of the reverse
// step's 15 us at 1024x256): every value as three integers over the block's largest
// exponent, whose sums over 128 threads are exact -- 2^-72 of the largest term.
// Infinities, NaNs and blocks below 2^-86 take the FP64 tree.
struct IntSums {
  unsigned top;
  int a, b, c;
};
__device__ __forceinline__ double block_sum(float v, double *sh, IntSums &is) {
  const int tid = threadIdx.y * ABX + threadIdx.x;
  // (is was cleared, and a barrier passed, by the caller)
  const unsigned m = __reduce_max_sync(0xffffffffu, __float_as_uint(v) & 0x7FFFFFFFu);
  if ((tid & 31) == 0) atomicMax(&is.top, m);
  __syncthreads();
  const int e = (int)(is.top >> 23);
  if (is.top == 0u) return 0.0;
  if (e < 40 || e == 255) return block_sum((double)v, sh);
  const FloatLimbs l = float_limbs(v, __uint_as_float((unsigned)(276 - e) << 23));
  const int sa = __reduce_add_sync(0xffffffffu, l.a), sb = __reduce_add_sync(0xffffffffu, l.b),
            sc = __reduce_add_sync(0xffffffffu, l.c);
  if ((tid & 31) == 0) {
    atomicAdd(&is.a, sa);
    atomicAdd(&is.b, sb);
    atomicAdd(&is.c, sc);
  }
  __syncthreads();
  if (tid != 0) return 0.0;
  constexpr double D = 1.0 / 16777216.0;
  return ((double)is.a + ((double)is.b + (double)is.c * D) * D) *
         __hiloint2double((1023 + e - 149) << 20, 0);
}
__device__ __forceinline__ double block_sum(double v, double *sh, IntSums &) {
  return block_sum(v, sh);
}

// One reverse step.  Bound by L2 and latency at the differentiation size (1024x256
// FP32: 124 bytes per cell, 32 MB).
// Measured, 600 steps of 1024x256 FP32 reversed and recomputed: 11.5 -> 6.5 ms; 10
// blocks per SM (6 in FP64) against the compiler's choice: 997x252 FP32 8.50 -> 8.44,
// 380x110 FP64 4.16 -> 4.08 ms for the whole call.
template <class A, bool FINAL>
__global__ void __launch_bounds__(ANT, sizeof(A) == 4 ? 10 : 6) adjoint_kernel(const AdjArgs a) {
  __shared__ double sh[ANT / 32];
  __shared__ IntSums is;
  const int nx = a.L.nx, ny = a.L.ny;
  const int x = blockIdx.x * ABX + threadIdx.x;
  const int y = blockIdx.y * ABY + threadIdx.y;
  const bool in = x < nx && y < ny;
  const long long N = (long long)nx * ny;
  const long long cell = (long long)y * nx + x;
  // Ahead of the predecessor's end (programmatic dependent launch): tables only.
  // Irregular cells take all their indices here, so that their loads are one round
  // like a regular cell's (reading the lists population by population made the
  // few irregular warps the whole launch's length: 17 us per step at 1024x256).
  const int aux = in ? a.aux[cell] : AUX_SOLID;
  unsigned lk = 0u, gw[3], pw[3];
  if (aux >= 0) {
    lk = a.lkr[aux];
#pragma unroll
    for (int w = 0; w < 3; ++w) {
      gw[w] = a.gat[(long long)w * a.nirr + aux];
      if constexpr (!FINAL) pw[w] = a.pul[(long long)w * a.nirr + aux];
    }
  }
  auto code = [](const unsigned *w, int j) { return (w[j / 4] >> (8 * (j % 4))) & 0xFFu; };
  // dense index of a contribution, storage index of a source
  auto row = [&](unsigned c) {
    int yy = y + (int)((c >> 2) & 3u) - 1;
    return yy < 0 ? yy + ny : yy >= ny ? yy - ny : yy;
  };
  auto dense = [&](unsigned c) {
    return (long long)(c >> 4) * N + (long long)row(c) * nx + x + (int)(c & 3u) - 1;
  };
  auto stored = [&](unsigned c) {
    return (long long)(c >> 4) * a.L.S + a.L.idx(x + (int)(c & 3u) - 1, row(c), 0);
  };
  A al = A(0);
  if constexpr (!FINAL)
    if (a.alpha && aux != AUX_SOLID) al = A(a.alpha[cell]);
  if (threadIdx.x == 0 && threadIdx.y == 0) is = {0u, 0, 0, 0};
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const A *mu_n = static_cast<const A *>(a.mu_next);
  const A *s = static_cast<const A *>(a.s);
  A *ga = static_cast<A *>(a.g_alpha);

  // lambda_{t+1}(X) = (P^T mu^{t+2})(X) + c_{t+1} dF/ds_{t+1}(X), and (not FINAL)
  // g_{t+1}(X) = (P s_t)(X).  Regular cells: plain shifts.  Irregular cells (box
  // faces, next to the body): the lists of contributing (Y, i) and of pull sources.
  // Every load of a path is issued before any is used.
  A lam[9], g[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) lam[k] = g[k] = A(0);
  A gacc = A(0);
  double *gb = a.g_block + 2 * ((long long)blockIdx.y * gridDim.x + blockIdx.x);
  double gb0 = 0.0;
  if constexpr (!FINAL)
    if (threadIdx.x == 0 && threadIdx.y == 0) gb0 = gb[0];
  int inl = 0;  // bit i: population i of g comes from the inlet
  if (aux == AUX_REGULAR) {
#pragma unroll
    for (int j = 0; j < 9; ++j) lam[j] = mu_n[j * N + cell + (long long)AYf(j) * nx + AXf(j)];
    if constexpr (!FINAL) {
      const long long c = a.L.idx(x, y, 0);
#pragma unroll
      for (int i = 0; i < 9; ++i) g[i] = s[i * a.L.S + c - a.L.off(AXf(i), AYf(i), 0)];
      gacc = ga[cell];
    }
  } else if (aux >= 0) {
#pragma unroll
    for (int j = 0; j < 9; ++j) {
      const unsigned c = code(gw, j);
      if (c != CODE_NONE) lam[j] = mu_n[dense(c)];
    }
    if constexpr (!FINAL) {
#pragma unroll
      for (int i = 0; i < 9; ++i) {
        const unsigned c = code(pw, i);
        if (c < CODE_INLET) g[i] = s[stored(c)];
      }
      gacc = ga[cell];
#pragma unroll
      for (int i = 0; i < 9; ++i) {
        const unsigned c = code(pw, i);
        if (c >= CODE_INLET) {
          if constexpr (sizeof(A) == 4) g[i] = a.fin_f[c - CODE_INLET];
          else g[i] = a.fin[c - CODE_INLET];
          inl |= 1 << i;
        }
      }
    }
    if (lk >> 31)  // further contributions
      for (int m = 1; m < GMAX; ++m) {
#pragma unroll
        for (int w = 0; w < 3; ++w) gw[w] = a.gat[(long long)(3 * m + w) * a.nirr + aux];
#pragma unroll
        for (int j = 0; j < 9; ++j) {
          const unsigned c = code(gw, j);
          if (c != CODE_NONE) lam[j] += mu_n[dense(c)];
        }
      }
    lk &= 0x7FFFFFFFu;
    if (lk) {
      // The segment index lives on the device so one captured graph reverses any
      // full segment: a launch reads k and the weight of its step t + 1.
      const A c2 =
          A(2.0 * (a.seg ? a.c_tab[(long long)(*a.seg) * a.K + 2 + a.q] : a.c_next));
#pragma unroll
      for (int j = 1; j < 9; ++j)
        if ((lk >> AOPPf(j)) & 1u) {
          const int e = a.obj_axis == 0 ? AXf(j) : AYf(j);
          if (e != 0) lam[j] += e > 0 ? c2 : -c2;
        }
    }
  }
  asm volatile("griddepcontrol.launch_dependents;");
  if constexpr (FINAL) {
    if (in) {
#pragma unroll
      for (int k = 0; k < 9; ++k) static_cast<A *>(a.mu_out)[k * N + cell] = lam[k];
    }
    return;
  } else {
    double d_u = 0.0;
    A dom = A(0);
    if (aux != AUX_SOLID) {
      // ---- mu = C'(g)^T lambda and the collision sensitivities -------------------
      const A one_a = A(1) - al, om = A(a.omega);
      A mu[9], jx, jy, vx, vy;
      if constexpr (sizeof(A) == 4) {
        // Population by population.  (Written with the forward sweep's conserving
        // constants the FP32 gradients come out 4 to 8 times nearer to FP64 on most
        // fields, but further off on the few where the rounding of the weights
        // happens to cancel the forward run's.)
        A rho3 = A(0);
        jx = jy = A(0);
#pragma unroll
        for (int i = 0; i < 9; ++i) {
          rho3 += g[i];
          if (AXf(i) != 0) jx += AXf(i) > 0 ? g[i] : -g[i];
          if (AYf(i) != 0) jy += AYf(i) > 0 ? g[i] : -g[i];
        }
        const A bx = one_a * jx, by = one_a * jy;
        const A usq = bx * bx + by * by;
        A A0 = A(0), A1x = A(0), A1y = A(0), A2x = A(0), A2y = A(0);
#pragma unroll
        for (int k = 0; k < 9; ++k) {
          const A w = A(aw(k));
          const A ex = AXf(k) == 0 ? A(0) : AXf(k) > 0 ? bx : -bx;
          const A ey = AYf(k) == 0 ? A(0) : AYf(k) > 0 ? by : -by;
          const A eu = AXf(k) == 0 ? ey : AYf(k) == 0 ? ex : ex + ey;
          const A feq = k == 0 ? w * (rho3 - A(1.5) * usq)
                               : w * (rho3 + A(3) * eu + A(4.5) * eu * eu - A(1.5) * usq);
          dom += lam[k] * (feq - g[k]);
          const A lw = lam[k] * w, lwe = lw * eu;
          A0 += lw;
          if (AXf(k) != 0) {
            A1x += AXf(k) > 0 ? lw : -lw;
            A2x += AXf(k) > 0 ? lwe : -lwe;
          }
          if (AYf(k) != 0) {
            A1y += AYf(k) > 0 ? lw : -lw;
            A2y += AYf(k) > 0 ? lwe : -lwe;
          }
        }
        vx = A(3) * A1x + A(9) * A2x - A(3) * bx * A0;
        vy = A(3) * A1y + A(9) * A2y - A(3) * by * A0;
#pragma unroll
        for (int i = 0; i < 9; ++i) {
          const A px = AXf(i) == 0 ? A(0) : AXf(i) > 0 ? vx : -vx;
          const A py = AYf(i) == 0 ? A(0) : AYf(i) > 0 ? vy : -vy;
          const A ve = AXf(i) == 0 ? py : AYf(i) == 0 ? px : px + py;
          mu[i] = (A(1) - om) * lam[i] + om * (i == 0 ? A0 : A0 + one_a * ve);
        }
      } else {
        // Over the +/- pairs: 130 FP64 operations, the pipe that binds here, for 310.
        constexpr A w0 = A(4.0 / 9.0), w1 = A(1.0 / 9.0), w2 = A(1.0 / 36.0);
        const A rho3 = g[0] + ((g[1] + g[3]) + (g[2] + g[4])) + ((g[5] + g[7]) + (g[6] + g[8]));
        jx = (g[1] - g[3]) + ((g[5] - g[7]) + (g[8] - g[6]));
        jy = (g[2] - g[4]) + ((g[5] - g[7]) + (g[6] - g[8]));
        const A bx = one_a * jx, by = one_a * jy;
        const A c0 = rho3 - A(1.5) * (bx * bx + by * by);
        const A bp = bx + by, bm = by - bx;  // e.u of populations 5 and 6
        dom = lam[0] * (w0 * c0 - g[0]);
        auto pair = [&](int i, int j, A w, A eu) {  // lambda (feq - g) of i and its opposite j
          const A ev = c0 + A(4.5) * (eu * eu);
          dom += lam[i] * (w * (ev + A(3) * eu) - g[i]);
          dom += lam[j] * (w * (ev - A(3) * eu) - g[j]);
        };
        pair(1, 3, w1, bx);
        pair(2, 4, w1, by);
        pair(5, 7, w2, bp);
        pair(6, 8, w2, bm);
        const A s1 = lam[1] + lam[3], s2 = lam[2] + lam[4], s5 = lam[5] + lam[7],
                s6 = lam[6] + lam[8];
        const A d1 = lam[1] - lam[3], d2 = lam[2] - lam[4], d5 = lam[5] - lam[7],
                d6 = lam[6] - lam[8];
        const A A0 = w0 * lam[0] + w1 * (s1 + s2) + w2 * (s5 + s6);
        const A A1x = w1 * d1 + w2 * (d5 - d6), A1y = w1 * d2 + w2 * (d5 + d6);
        const A A2x = w1 * (s1 * bx) + w2 * (s5 * bp - s6 * bm);
        const A A2y = w1 * (s2 * by) + w2 * (s5 * bp + s6 * bm);
        vx = A(3) * A1x + A(9) * A2x - A(3) * (bx * A0);
        vy = A(3) * A1y + A(9) * A2y - A(3) * (by * A0);
        const A omc = A(1) - om, P = om * A0, qx = om * (one_a * vx), qy = om * (one_a * vy);
        const A qp = qx + qy, qm = qy - qx;
        const A add[9] = {P, P + qx, P + qy, P - qx, P - qy, P + qp, P + qm, P - qp, P - qm};
#pragma unroll
        for (int i = 0; i < 9; ++i) mu[i] = omc * lam[i] + add[i];
      }
      if (inl) {
#pragma unroll
        for (int i = 0; i < 9; ++i)
          if ((inl >> i) & 1)
            d_u += static_cast<double>(mu[i]) *
                   a.dfin[code(pw, i) - CODE_INLET];
      }
      // d feq / d alpha, with d u_B / d alpha = -(jx, jy).
      ga[cell] = gacc - om * (vx * jx + vy * jy);
#pragma unroll
      for (int k = 0; k < 9; ++k) static_cast<A *>(a.mu_out)[k * N + cell] = mu[k];
    }
    // the inlet is the column x = 0: lane 0 of a warp
    __shared__ double shu[ABY];
    if (x == 0) shu[threadIdx.y] = d_u;
    __syncthreads();
    const double so = block_sum(dom, sh, is);
    if (threadIdx.x == 0 && threadIdx.y == 0) {
      gb[0] = gb0 + so;
      if (x == 0) {
        double su = 0.0;
        for (int w = 0; w < ABY; ++w) su += shu[w];
        gb[1] += su;
      }
    }
  }
}

// Sensitivities of the initial state s_1 = C(feq(U0)) through lambda_1:
// U0 = (u_in, v0) in fluid cells, U_B = (1 - alpha) U0, p = 0.
template <class A>
__global__ void __launch_bounds__(ANT) init_sens_kernel(const AdjArgs a, const A *lam1,
                                                        unsigned long long seed, double amp,
                                                        double *g_alpha64) {
  __shared__ double sh[ANT / 32];
  const int nx = a.L.nx, ny = a.L.ny;
  const int x = blockIdx.x * ABX + threadIdx.x;
  const int y = blockIdx.y * ABY + threadIdx.y;
  const long long N = (long long)nx * ny;
  const long long cell = (long long)y * nx + x;
  double gu = 0.0, gom = 0.0;
  if (x < nx && y < ny && !mask_solid(a.mask, a.nxw, ny, x, y, 0)) {
    const double al = a.alpha ? (double)a.alpha[cell] : 0.0;
    const double ux = a.u_in, uy = perturbation(seed, cell, amp);
    const double bx = (1.0 - al) * ux, by = (1.0 - al) * uy;
    const double om = a.omega;
    double gal = 0.0;
    for (int k = 0; k < 9; ++k) {
      const double w = aw(k), ex = AXf(k), ey = AYf(k);
      const double eu = ex * ux + ey * uy, eb = ex * bx + ey * by;
      const double f0 = w * (3.0 * eu + 4.5 * eu * eu - 1.5 * (ux * ux + uy * uy));
      const double fb = w * (3.0 * eb + 4.5 * eb * eb - 1.5 * (bx * bx + by * by));
      const double df0 = w * (3.0 * ex + 9.0 * eu * ex - 3.0 * ux);
      const double dfb = (1.0 - al) * w * (3.0 * ex + 9.0 * eb * ex - 3.0 * bx);
      const double l = (double)lam1[k * N + cell];
      gu += l * ((1.0 - om) * df0 + om * dfb);
      gom += l * (fb - f0);
      gal += l * om * w * (-3.0 * eu - 9.0 * eb * eu + 3.0 * (bx * ux + by * uy));
    }
    g_alpha64[cell] += gal;
  }
  const double so = block_sum(gom, sh), su = block_sum(gu, sh);
  if (threadIdx.x == 0 && threadIdx.y == 0) {
    double *gb = a.g_block + 2 * ((long long)blockIdx.y * gridDim.x + blockIdx.x);
    gb[0] += so;
    gb[1] += su;
  }
}

// End of a checkpoint segment: g64 += gA; gA = 0; the segment index steps back
// (every kernel that reads it precedes this one on the stream).
template <class A>
__global__ void flush_kernel(A *ga, double *g64, long long n, int *seg) {
  for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < n;
       c += (long long)gridDim.x * blockDim.x) {
    g64[c] += static_cast<double>(ga[c]);
    ga[c] = A(0);
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) *seg -= 1;
}

// The recompute stream's segment index steps back after its segment.
__global__ void step_back_kernel(int *seg) { *seg -= 1; }

// seg_states[0] = checkpoint k = *seg (16-byte words; sizes are multiples of 16).
__global__ void checkpoint_copy_kernel(const uint4 *ck, const int *seg, long long words,
                                       uint4 *dst) {
  const uint4 *src = ck + (long long)(*seg) * words;
  for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < words;
       c += (long long)gridDim.x * blockDim.x)
    dst[c] = src[c];
}

int afail(int code, const std::string &m) { return record_error(code, m.c_str()); }

#define ACK(call)                                                                         \
  do {                                                                                    \
    cudaError_t e_ = (call);                                                              \
    if (e_ != cudaSuccess)                                                                \
      return afail(CFLBM_E_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_));     \
  } while (0)

// Device scratch of one adjoint run: arrays laid out in one allocation, freed on
// return.
struct AdjScratch {
  char *base = nullptr;
  size_t bytes = 0;
  std::vector<std::pair<void **, size_t>> parts;
  ~AdjScratch() {
    if (base) cudaFree(base);
  }
  template <class T>
  void add(T **p, size_t n) {
    parts.push_back({reinterpret_cast<void **>(p), bytes});
    bytes += (std::max<size_t>(n, 1) * sizeof(T) + 255) / 256 * 256;
  }
  cudaError_t alloc() {
    const cudaError_t e = cudaMalloc(&base, bytes);
    if (e != cudaSuccess) {
      base = nullptr;
      return e;
    }
    for (const auto &p : parts) *p.first = base + p.second;
    return cudaSuccess;
  }
};

// The second stream of the reverse sweep and its fork/join events.
struct AdjStreams {
  cudaStream_t rec = nullptr;
  cudaEvent_t fork = nullptr, join = nullptr;
  cudaError_t create() {
    cudaError_t e = cudaStreamCreateWithFlags(&rec, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&fork, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&join, cudaEventDisableTiming);
    return e;
  }
  ~AdjStreams() {
    if (rec) cudaStreamSynchronize(rec);
    if (fork) cudaEventDestroy(fork);
    if (join) cudaEventDestroy(join);
    if (rec) cudaStreamDestroy(rec);
  }
};

// Tables of the reverse sweep.  Every fluid cell X is classified from the forward
// pull itself: X is regular when its own pull is the plain shift (source X - e_i,
// population i, for every i) and the pulls that read X are exactly the 9 plain ones
// ((X + e_j, j) for every j) -- away from the box's faces, all 8 neighbours fluid.
// For every other fluid cell (box faces, cells next to the body) the entry lists,
// per population j of X, every pull (Y, i) whose source is (X, j), in the order of
// (Y, i), and X's own 9 pull sources; lkr holds its
// link bits (the momentum-exchange force reads them).  Entries are numbered as they
// come; counters: [0] entries, [1] more than GMAX pulls read one population.
__global__ void __launch_bounds__(ANT) classify_kernel(const uint32_t *mask, int nxw, int nx,
                                                       int ny, int *aux, int *counters) {
  const int x = blockIdx.x * ABX + threadIdx.x, y = blockIdx.y * ABY + threadIdx.y;
  if (x >= nx || y >= ny) return;
  int v = AUX_REGULAR;
  if (mask_solid(mask, nxw, ny, x, y, 0)) {
    v = AUX_SOLID;
  } else {
    bool irr = x == 0 || x == nx - 1 || y == 0 || y == ny - 1;
    for (int d = 0; d < 9 && !irr; ++d)
      irr = mask_solid(mask, nxw, ny, x + d % 3 - 1, y + d / 3 - 1, 0);
    if (irr) v = atomicAdd(&counters[0], 1);
  }
  aux[(long long)y * nx + x] = v;
}

__global__ void __launch_bounds__(ANT) tables_kernel(const Layout L, const uint32_t *mask,
                                                     int nxw, int wall_y, const int *aux,
                                                     long long nirr, unsigned *gat,
                                                     unsigned *pul, unsigned *lkr,
                                                     int *counters) {
  const int nx = L.nx, ny = L.ny;
  const int x = blockIdx.x * ABX + threadIdx.x, y = blockIdx.y * ABY + threadIdx.y;
  if (x >= nx || y >= ny) return;
  const int r = aux[(long long)y * nx + x];
  if (r < 0) return;
  const unsigned lk = link_bits(mask, nxw, nx, ny, wall_y, x, y);
  // (x, y) -> (xx, yy) in steps; a wrapped row is one step the other way
  auto step_y = [&](int yy) { return yy == y ? 0 : (yy == y + 1 || yy == y + 1 - ny) ? 1 : -1; };
  unsigned w[3] = {0u, 0u, 0u};
  for (int i = 0; i < 9; ++i) {
    int sx, sy, j;
    const int kind = pull_source(nx, ny, wall_y, lk, x, y, i, sx, sy, j);
    const unsigned c = kind == SRC_INLET ? CODE_INLET + j : cell_code(j, sx - x, step_y(sy));
    w[i / 4] |= c << (8 * (i % 4));
  }
  for (int k = 0; k < 3; ++k) pul[k * nirr + r] = w[k];
  unsigned gw[3 * GMAX];
  for (int k = 0; k < 3 * GMAX; ++k) gw[k] = ~0u;  // CODE_NONE
  int cnt[9] = {0};
  // the neighbouring rows in ascending order (periodic walls wrap)
  int rows[3], nr = 0;
  for (int d = -1; d <= 1; ++d) {
    int yy = y + d;
    if (yy < 0 || yy >= ny) {
      if (wall_y != WALL_PERIODIC) continue;
      yy = yy < 0 ? yy + ny : yy - ny;
    }
    int at = nr++;
    for (; at > 0 && rows[at - 1] > yy; --at) rows[at] = rows[at - 1];
    rows[at] = yy;
  }
  for (int k = 0; k < nr; ++k)
    for (int xx = max(x - 1, 0); xx <= min(x + 1, nx - 1); ++xx) {
      const int yy = rows[k];
      if (mask_solid(mask, nxw, ny, xx, yy, 0)) continue;
      const unsigned lY = link_bits(mask, nxw, nx, ny, wall_y, xx, yy);
      for (int i = 0; i < 9; ++i) {
        int sx, sy, j;
        if (pull_source(nx, ny, wall_y, lY, xx, yy, i, sx, sy, j) == SRC_INLET || sx != x || sy != y)
          continue;
        if (cnt[j] == GMAX) {
          counters[1] = 1;
          continue;
        }
        const unsigned c = cell_code(i, xx - x, step_y(yy)) ^ 0xFFu;
        gw[3 * cnt[j]++ + j / 4] ^= c << (8 * (j % 4));
      }
    }
  for (int k = 0; k < 3 * GMAX; ++k) gat[k * nirr + r] = gw[k];
  bool more = false;
  for (int j = 0; j < 9; ++j) more = more || cnt[j] > 1;
  lkr[r] = lk | (more ? 0x80000000u : 0u);
}

template <class A>
int run_adjoint(cflbm_handle *h, const cflbm_adjoint_spec *sp, double *dJ_dalpha,
                cflbm_adjoint_result *res) {
  using clk = std::chrono::steady_clock;
  const Layout &L = h->L;
  const int nx = L.nx, ny = L.ny;
  const long long N = (long long)nx * ny;
  const int T = sp->steps, K = sp->checkpoint_every;
  const size_t sb = h->f_bytes;
  const int nck = (T + K - 1) / K;
  const dim3 blk(ABX, ABY), grd((nx + ABX - 1) / ABX, (ny + ABY - 1) / ABY);
  const long long nblk = (long long)grd.x * grd.y;
  cudaStream_t st = h->stream;

  AdjScratch sc;
  char *ck = nullptr, *seg = nullptr;
  A *mu0 = nullptr, *mu1 = nullptr, *ga = nullptr;
  double *ga64 = nullptr, *gblk = nullptr, *c_tab = nullptr;
  int *aux = nullptr, *counters = nullptr, *d_seg = nullptr;
  unsigned *gat = nullptr, *pul = nullptr, *lkr = nullptr;
  // One block for all (a cudaMalloc and its cudaFree cost about 0.1 ms each).  What
  // starts at zero comes first: mu1, ga, ga64, gblk, counters.
  sc.add(&mu1, 9 * (size_t)N);
  sc.add(&ga, N);
  sc.add(&ga64, N);
  sc.add(&gblk, 2 * nblk);
  sc.add(&counters, 2);
  const size_t zeroed = sc.bytes;
  sc.add(&mu0, 9 * (size_t)N);
  sc.add(&aux, N);
  sc.add(&d_seg, 2);
  sc.add(&c_tab, (size_t)T + 2);
  sc.add(&ck, (size_t)nck * sb);
  sc.add(&seg, 2 * (size_t)K * sb);
  ACK(sc.alloc());
  ACK(cudaMemsetAsync(sc.base, 0, zeroed, st));
  classify_kernel<<<grd, blk, 0, st>>>(h->d_mask, h->nxw, nx, ny, aux, counters);
  ACK(cudaGetLastError());
  int cnt[2] = {0, 0};
  ACK(cudaMemcpyAsync(cnt, counters, sizeof(cnt), cudaMemcpyDeviceToHost, st));
  ACK(cudaStreamSynchronize(st));
  const long long n_irregular = cnt[0];
  AdjScratch st_tab;
  st_tab.add(&gat, (size_t)n_irregular * 3 * GMAX);
  st_tab.add(&pul, (size_t)n_irregular * 3);
  st_tab.add(&lkr, (size_t)n_irregular);
  ACK(st_tab.alloc());
  tables_kernel<<<grd, blk, 0, st>>>(L, h->d_mask, h->nxw, h->cfg.wall_y, aux, n_irregular, gat,
                                     pul, lkr, counters);
  count_launch(2);
  ACK(cudaGetLastError());
  ACK(cudaMemcpyAsync(cnt, counters, sizeof(cnt), cudaMemcpyDeviceToHost, st));
  ACK(cudaStreamSynchronize(st));
  if (cnt[1])
    return afail(CFLBM_E_UNSUPPORTED, "cflbm_adjoint: more than 4 pulls read one population");

  // ---- forward run, keeping s_1, s_{K+1}, s_{2K+1}, ... ---------------------------
  const auto t_f0 = clk::now();
  for (int k = 0; k < nck; ++k) {
    ACK(cudaMemcpyAsync(ck + (size_t)k * sb, h->fA, sb, cudaMemcpyDeviceToDevice, st));
    int rc = cflbm_step(h, std::min(K, T - k * K));
    if (rc) return rc;
  }
  ACK(cudaStreamSynchronize(st));
  const double t_forward = std::chrono::duration<double>(clk::now() - t_f0).count();
  std::vector<double> hist(3 * (size_t)T);
  int64_t nh = 0;
  int rc = cflbm_force_history(h, hist.data(), T, &nh);
  if (rc) return rc;
  if (nh != T) return afail(CFLBM_E_INVALID, "cflbm_adjoint: force history shorter than the run");
  const int t0 = sp->window_begin, t1 = sp->window_end;
  const double cw = 1.0 / (t1 - t0 + 1);
  double J = 0.0;
  for (int t = t0; t <= t1; ++t) J += cw * hist[3 * (size_t)(t - 1) + sp->objective];

  // ---- reverse sweep, one checkpoint segment at a time ----------------------------
  // Segment k holds states s_{kK+1} .. s_{kK+n}.  Recomputing it (copy
  // checkpoint k, n - 1 forward sweeps) and reversing it (adjoint kernels from
  // the top state down, then the flush) use one of two state buffers, k % 2.
  // Unit k reverses segment k on the main stream while a second stream
  // recomputes segment k - 1 into the other buffer; the unit joins at its end.
  // The segment indices the kernels read are device integers (one for each
  // stream's work, stepped by the stream's last kernel), so every interior unit
  // is the same launch sequence: it is captured as a CUDA graph per buffer and
  // mu parity and replayed.  The first unit (partial top segment, whose top
  // state s_T has lambda_{T+1} = 0) and the last (nothing left to recompute)
  // run as direct launches.
  const auto t_r0 = clk::now();
  {  // d_seg[0]: segment being reversed, [1]: segment being recomputed
    std::vector<double> ct((size_t)T + 2, 0.0);
    for (int t = t0; t <= t1; ++t) ct[t] = cw;
    const int k_last[2] = {nck - 1, nck - 1};
    ACK(cudaMemcpyAsync(c_tab, ct.data(), ct.size() * 8, cudaMemcpyHostToDevice, st));
    ACK(cudaMemcpyAsync(d_seg, k_last, 8, cudaMemcpyHostToDevice, st));
    ACK(cudaStreamSynchronize(st));
  }
  AdjStreams rs;
  ACK(rs.create());
  cudaStream_t rec = rs.rec;
  AdjArgs aa{};
  aa.L = L;
  aa.mask = h->d_mask;
  aa.nxw = h->nxw;
  aa.aux = aux;
  aa.gat = gat;
  aa.pul = pul;
  aa.lkr = lkr;
  aa.nirr = (int)n_irregular;
  aa.alpha = h->d_alpha;
  aa.omega = h->omega;
  aa.u_in = h->cfg.u0;
  for (int j = 0; j < 9; ++j) {
    aa.fin[j] = inlet_f(j, h->cfg.u0);
    aa.fin_f[j] = (float)aa.fin[j];
    aa.dfin[j] = inlet_dfdu(j, h->cfg.u0);
  }
  aa.obj_axis = sp->objective;
  aa.g_alpha = ga;
  aa.g_block = gblk;
  aa.seg = d_seg;
  aa.c_tab = c_tab;
  aa.K = K;
  A *mu_next = mu1, *mu_cur = mu0;
  const long long words = (long long)(sb / 16);
  const int copy_blocks = (int)std::min<long long>((words + 255) / 256, 4096);
  const int flush_blocks = (int)std::min<long long>((N + 255) / 256, 4096);
  char *buf[2] = {seg, seg + (size_t)K * sb};
  // Recompute one segment of n states into b (stream s).
  auto recompute = [&](cudaStream_t s, char *b, int n) -> int {
    checkpoint_copy_kernel<<<copy_blocks, 256, 0, s>>>(reinterpret_cast<const uint4 *>(ck),
                                                        d_seg + 1, words,
                                                        reinterpret_cast<uint4 *>(b));
    for (int q = 1; q < n; ++q) {
      SweepArgs sa = channel_args(h, b + (size_t)(q - 1) * sb, b + (size_t)q * sb, false);
      sa.bnd_blocks = 0;  // the force of these steps is known
      ACK(launch_sweep_channel(9, h->cfg.storage, h->cfg.compute, sa, s));
    }
    step_back_kernel<<<1, 1, 0, s>>>(d_seg + 1);
    count_launch(2);
    ACK(cudaGetLastError());
    return CFLBM_OK;
  };
  // Reverse one segment of n states held in b (main stream).
  auto reverse = [&](char *b, int n, bool skip_top) -> int {
    bool chained = false;
    for (int q = n - 1; q >= 0; --q) {
      if (skip_top && q == n - 1) continue;
      aa.s = b + (size_t)q * sb;
      aa.q = q;
      aa.mu_next = mu_next;
      aa.mu_out = mu_cur;
      // chained to the reverse step before it; the unit's first one also waits for
      // the other stream and starts plainly
      cudaLaunchAttribute at{};
      at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
      at.val.programmaticStreamSerializationAllowed = 1;
      cudaLaunchConfig_t lc{};
      lc.gridDim = grd;
      lc.blockDim = blk;
      lc.stream = st;
      lc.attrs = &at;
      lc.numAttrs = chained ? 1 : 0;
      ACK(cudaLaunchKernelEx(&lc, adjoint_kernel<A, false>, aa));
      chained = true;
      count_launch(1);
      std::swap(mu_next, mu_cur);
    }
    flush_kernel<A><<<flush_blocks, 256, 0, st>>>(ga, ga64, N, d_seg);
    count_launch(1);
    ACK(cudaGetLastError());
    return CFLBM_OK;
  };
  // Unit k: reverse segment k (n states, buffer k % 2) while recomputing
  // segment k - 1 (K states, the other buffer) when k > 0.
  auto unit = [&](int k, int n, bool skip_top) -> int {
    ACK(cudaEventRecord(rs.fork, st));
    ACK(cudaStreamWaitEvent(rec, rs.fork, 0));
    if (k > 0) {
      const int rc2 = recompute(rec, buf[(k - 1) & 1], K);
      if (rc2) return rc2;
    }
    const int rc1 = reverse(buf[k & 1], n, skip_top);
    if (rc1) return rc1;
    ACK(cudaEventRecord(rs.join, rec));
    ACK(cudaStreamWaitEvent(st, rs.join, 0));
    return CFLBM_OK;
  };
  const int n_top = T - (nck - 1) * K;
  int urc = recompute(st, buf[(nck - 1) & 1], n_top);
  if (!urc) urc = unit(nck - 1, n_top, true);
  if (urc) return urc;
  cudaGraphExec_t gexec[4] = {nullptr, nullptr, nullptr, nullptr};
  struct GraphGuard {
    cudaGraphExec_t *g;
    ~GraphGuard() {
      for (int i = 0; i < 4; ++i)
        if (g[i]) cudaGraphExecDestroy(g[i]);
    }
  } guard{gexec};
  long long graph_launches = 0;
  for (int k = nck - 2; k >= 1; --k) {
    const int gi = (k & 1) * 2 + (mu_next == mu1 ? 0 : 1);
    if (nck - 2 < GRAPH_UNITS) {
      if ((urc = unit(k, K, false))) return urc;
    } else if (!gexec[gi]) {
      const long long n0 = cflbm_launch_count();
      cudaGraph_t g = nullptr;
      ACK(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
      const int rcs = unit(k, K, false);
      const cudaError_t ec = cudaStreamEndCapture(st, &g);
      if (rcs) {
        if (g) cudaGraphDestroy(g);
        return rcs;
      }
      ACK(ec);
      const cudaError_t ei = cudaGraphInstantiate(&gexec[gi], g, 0);
      cudaGraphDestroy(g);
      ACK(ei);
      graph_launches = cflbm_launch_count() - n0;
      // Capture counted the launches and moved the host-side mu parity; this
      // first replay runs them.
      ACK(cudaGraphLaunch(gexec[gi], st));
    } else {
      ACK(cudaGraphLaunch(gexec[gi], st));
      count_launch(graph_launches);
      if (K & 1) std::swap(mu_next, mu_cur);
    }
  }
  if (nck >= 2) {
    urc = unit(0, K, false);
    if (urc) return urc;
  }
  // lambda_1 and the sensitivities of the initial state.
  aa.mu_next = mu_next;
  aa.mu_out = mu_cur;
  aa.seg = nullptr;
  aa.c_next = (1 >= t0 && 1 <= t1) ? cw : 0.0;
  adjoint_kernel<A, true><<<grd, blk, 0, st>>>(aa);
  init_sens_kernel<A><<<grd, blk, 0, st>>>(aa, mu_cur, h->cfg.seed, h->cfg.perturb_amp, ga64);
  count_launch(2);
  ACK(cudaGetLastError());
  std::vector<double> hgb(2 * nblk);
  if (dJ_dalpha) ACK(cudaMemcpyAsync(dJ_dalpha, ga64, N * 8, cudaMemcpyDeviceToHost, st));
  ACK(cudaMemcpyAsync(hgb.data(), gblk, 2 * nblk * 8, cudaMemcpyDeviceToHost, st));
  ACK(cudaStreamSynchronize(st));
  const double t_reverse = std::chrono::duration<double>(clk::now() - t_r0).count();
  double somega = 0.0, su = 0.0;
  for (long long b = 0; b < nblk; ++b) {
    somega += hgb[2 * b];
    su += hgb[2 * b + 1];
  }
  std::memset(res, 0, sizeof(*res));
  res->J = J;
  res->dJ_du_in = su;
  res->dJ_dtau = -h->omega * h->omega * somega;
  res->seconds_forward = t_forward;
  res->seconds_reverse = t_reverse;
  res->device_bytes = (int64_t)((size_t)(nck + 2 * K) * sb + (2 * 9 + 1) * N * sizeof(A) +
                                N * (8 + 4) + n_irregular * (3 * GMAX + 3 + 1) * 4 +
                                2 * nblk * 8);
  return CFLBM_OK;
}

}  // namespace

extern "C" int cflbm_adjoint(cflbm_handle *h, const cflbm_adjoint_spec *sp, double *dJ_dalpha,
                             cflbm_adjoint_result *res) {
  if (!h || !sp || !res) return afail(CFLBM_E_INVALID, "cflbm_adjoint: null argument");
  if (h->Q != 9 || h->cfg.profile != CFLBM_PROFILE_CHANNEL)
    return afail(CFLBM_E_UNSUPPORTED, "cflbm_adjoint: the adjoint covers the D2Q9 channel profile");
  const bool f32 = h->cfg.storage == CFLBM_STORE_FP32 && h->cfg.compute == CFLBM_COMPUTE_FP32;
  const bool f64 = h->cfg.storage == CFLBM_STORE_FP64 && h->cfg.compute == CFLBM_COMPUTE_FP64;
  if (!f32 && !f64)
    return afail(CFLBM_E_UNSUPPORTED,
                 "cflbm_adjoint: storage/arithmetic must be FP32/FP32 or FP64/FP64");
  if (h->batched) return afail(CFLBM_E_INVALID, "cflbm_adjoint: batch instances are not supported");
  if (h->steps_done != 0) return afail(CFLBM_E_INVALID, "cflbm_adjoint: needs a fresh handle");
  if (h->L.nx < 3 || h->L.ny < 3)
    return afail(CFLBM_E_INVALID, "cflbm_adjoint: needs nx, ny >= 3");
  if (sp->steps < 1 || sp->checkpoint_every < 1 || sp->window_begin < 1 ||
      sp->window_end < sp->window_begin || sp->window_end > sp->steps ||
      (sp->objective != 0 && sp->objective != 1))
    return afail(CFLBM_E_INVALID, "cflbm_adjoint: bad spec (steps, checkpoint, window, objective)");
  if (h->hist_cap < sp->steps)
    return afail(CFLBM_E_INVALID, "cflbm_adjoint: force_history must hold every step of the run");
  cudaError_t e = cudaSetDevice(h->cfg.device);
  if (e != cudaSuccess) return afail(CFLBM_E_CUDA, cudaGetErrorString(e));
  return f32 ? run_adjoint<float>(h, sp, dJ_dalpha, res)
             : run_adjoint<double>(h, sp, dJ_dalpha, res);
}

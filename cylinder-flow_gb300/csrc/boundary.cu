// Boundary, bounce-back/force, initialisation and reduction kernels.
//
// These run on O(surface) work (ghost layers, fluid->solid links) except the
// initialisation, reduction and dump/restore kernels, which run once or on
// demand.  The hot per-step sweep is in sweep.cuh.
#include "fixed.cuh"
#include "solver.cuh"

namespace cflbm {

namespace {

long long g_launches = 0;

// Runtime direction tables (boundary kernels index directions dynamically).
template <int Q> struct DT;
__constant__ signed char c_e9[9][2] = {{0, 0}, {1, 0},  {0, 1},   {-1, 0}, {0, -1},
                                        {1, 1}, {-1, 1}, {-1, -1}, {1, -1}};
template <> struct DT<9> {
  __device__ static int ex(int i) { return c_e9[i][0]; }
  __device__ static int ey(int i) { return c_e9[i][1]; }
  __device__ static int ez(int) { return 0; }
};
__constant__ signed char c_e27[27][3] = {
    {0, 0, 0},  {1, 0, 0},   {-1, 0, 0}, {0, 1, 0},   {0, -1, 0},  {0, 0, 1},   {0, 0, -1},
    {1, 1, 0},  {-1, -1, 0}, {1, -1, 0}, {-1, 1, 0},  {1, 0, 1},   {-1, 0, -1}, {1, 0, -1},
    {-1, 0, 1}, {0, 1, 1},   {0, -1, -1}, {0, 1, -1}, {0, -1, 1},  {1, 1, 1},   {-1, -1, -1},
    {1, -1, 1}, {-1, 1, -1}, {1, 1, -1}, {-1, -1, 1}, {1, -1, -1}, {-1, 1, 1}};
template <> struct DT<27> {
  __device__ static int ex(int i) { return c_e27[i][0]; }
  __device__ static int ey(int i) { return c_e27[i][1]; }
  __device__ static int ez(int i) { return c_e27[i][2]; }
};
template <int Q> __device__ int dopp(int i) { return Lat<Q>::opp(i); }
// D2Q9 opposite for a run-time index, without a table in local memory:
// 1<->3, 2<->4 (axes), 5<->7, 6<->8 (diagonals).
template <> __device__ int dopp<9>(int i) {
  return i == 0 ? 0 : (i <= 4 ? (i + 1) % 4 + 1 : (i - 3) % 4 + 5);
}
// FP64 values of stored elements and back (Store<> codecs; L.fbase is the
// FP16 format's storage offset per population).
template <class ST> struct Dec;
template <> struct Dec<double> {
  template <int Q> __device__ static double get(double v, int, const Layout &) { return v; }
  template <int Q> __device__ static double put(double v, int, const Layout &) { return v; }
};
template <> struct Dec<float> {
  template <int Q> __device__ static double get(float v, int, const Layout &) {
    return (double)v;
  }
  template <int Q> __device__ static float put(double v, int, const Layout &) {
    return (float)v;
  }
};
template <> struct Dec<F16Dev> {
  template <int Q> __device__ static double get(__half v, int i, const Layout &L) {
    return __fma_rn((double)__half2float(v), 1.0 / F16_SCALE, (double)L.fbase[i]);
  }
  template <int Q> __device__ static __half put(double v, int i, const Layout &L) {
    return __double2half(__dmul_rn(__dsub_rn(v, (double)L.fbase[i]), (double)F16_SCALE));
  }
};

inline int blocks_for(long long n, int threads) {
  long long b = (n + threads - 1) / threads;
  if (b < 1) b = 1;
  if (b > 65535LL * 8) b = 65535LL * 8;
  return (int)b;
}

// ---- solid links: bounce-back fill + momentum-exchange force ----------------
// For link (s, k): s solid, X = s + e_k fluid.  Fill f_k(s) = f*_{opp(k)}(s +
// reach*e_k) (reach 1: halfway bounce-back; reach 2: the reference's usrbc,
// "3D.../lbm.cpp:350-356", "MPI Kokkos/lbm.cpp:347-353").  Force: the reference's
// momentum exchange ("MPI Kokkos/lbm.cpp:364-377") sums, over fluid X and
// direction ii = opp(k) pointing into the solid, (f_ii(X) + f_opp(ii)(X + e_ii))
// e_ii after the fill.  Reduced per block in FP64, then by the last of a.blocks
// blocks in block order (deterministic), into the force history slot of this step.
template <int Q, class ST>
__device__ __forceinline__ void links_block(const LinkArgs &a) {
  using E = typename Store<ST>::elem;
  E *f = static_cast<E *>(a.f);
  const Layout &L = a.L;
  double s[3] = {0.0, 0.0, 0.0};
  long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  int4 l = make_int4(0, 0, 0, 0);
  if (t < a.n) l = a.links[t];
  asm volatile("griddepcontrol.wait;" ::: "memory");
  while (t < a.n) {
    const int k = l.w, kb = dopp<Q>(k);
    const long long ok = L.off(DT<Q>::ex(k), DT<Q>::ey(k), DT<Q>::ez(k));
    const long long c = L.idx(l.x, l.y, l.z);
    const E v = f[kb * L.S + c + a.reach * ok];
    f[k * L.S + c] = v;
    const double m = Dec<ST>::template get<Q>(f[kb * L.S + c + ok], kb, L) +
                     Dec<ST>::template get<Q>(v, kb, L);
    s[0] += m * DT<Q>::ex(kb);
    s[1] += m * DT<Q>::ey(kb);
    s[2] += m * DT<Q>::ez(kb);
    t += (long long)a.blocks * blockDim.x;
    if (t < a.n) l = a.links[t];
  }
  __shared__ double sh[3][8];
  __shared__ bool last;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  auto block_sums = [&] {  // valid in thread 0
    for (int o = 16; o > 0; o >>= 1)
      for (int d = 0; d < 3; ++d) s[d] += __shfl_down_sync(0xffffffffu, s[d], o);
    if (lane == 0)
      for (int d = 0; d < 3; ++d) sh[d][wid] = s[d];
    __syncthreads();
    if (threadIdx.x == 0)
      for (int d = 0; d < 3; ++d) {
        s[d] = 0.0;
        for (int w = 0; w < 8; ++w) s[d] += sh[d][w];
      }
  };
  auto record = [&] {
    const long long st = *a.step;
    for (int d = 0; d < 3; ++d) a.hist[3 * (st % a.cap) + d] = s[d];
    *a.step = st + 1;
  };
  block_sums();
  if (a.blocks == 1) {
    if (threadIdx.x == 0) record();
    return;
  }
  if (threadIdx.x == 0) {
    for (int d = 0; d < 3; ++d) a.partials[3 * blockIdx.x + d] = s[d];
    __threadfence();
    last = (atomicAdd(a.counter, 1u) == (unsigned)a.blocks - 1);
  }
  __syncthreads();
  if (last) {
    __threadfence();
    const volatile double *p = a.partials;
    for (int d = 0; d < 3; ++d) s[d] = 0.0;
    for (int b = threadIdx.x; b < a.blocks; b += blockDim.x)
      for (int d = 0; d < 3; ++d) s[d] += p[3 * b + d];
    __syncthreads();
    block_sums();
    if (threadIdx.x == 0) {
      record();
      *a.counter = 0u;
    }
  }
}

// ---- reference-profile boundary launch ------------------------------------------
// One pass of the reference's Streaming() boundary sequence over a face:
//   copy   (x low,  e_x > 0): f_i(-1, j, k)  = f_i(0, j, k)
//          ("3D MPI+KOKKOS+MPIIO/lbm.cpp:326-335", "MPI Kokkos/lbm.cpp:315-321")
//   extrap (x high, e_x < 0): f_i(nx, j, k) = f_i(nx-1, j+e_y, k+e_z)    (:338-347, :323-329)
//   bounce (wall, e_a pointing inward): the ghost layer takes the opposite
//          population two layers in, shifted by twice the in-plane velocity
//          (:278-324, :331-345).
// Tangential ranges cover the interior plus one ring, [-1, n+1), as the
// reference's [ghost-1, l-ghost+1).
// All passes of a step run as one launch, one thread per (pass, population, face
// cell), and the link fill with them where no solid cell is within two cells of a
// face (then neither reads what the other writes).  The passes' order lives in
// the reads: a source in a ghost layer that an earlier pass of the step writes is
// followed to that pass's own source, until it is an interior cell or a ghost that
// no earlier pass has written.  Such a ghost holds the step before's value, which the
// other buffer has (its ghosts were filled for the step before, and ghosts that no
// pass writes are the same in both), so nothing written here is read here.
// Measured, REF3D 257x97x97 FP64, 20 steps and the fields: 5.01 ms against 5.51 ms
// with three launches of two passes each and one for the links; REF2D 266x174, 50
// steps: 0.33 ms against 1.06 ms.
struct PassCell {
  int c[3];
};
// The source of pass op for population i at ghost cell g, and its population.
template <int Q>
__device__ __forceinline__ PassCell pass_source(const FaceOp &op, const int *n, PassCell g, int &i) {
  const int e[3] = {DT<Q>::ex(i), DT<Q>::ey(i), DT<Q>::ez(i)};
  const int f = op.kind == 0 ? 0 : op.kind == 1 ? 1 : 2;  // in-plane shift in e
#pragma unroll
  for (int d = 0; d < 3; ++d) g.c[d] += d == op.axis ? 0 : f * e[d];
  const int v = op.kind == 0 ? 0 : op.kind == 1 ? n[0] - 1 : op.side == 0 ? 1 : n[op.axis] - 2;
#pragma unroll
  for (int d = 0; d < 3; ++d)
    if (d == op.axis) g.c[d] = v;
  if (op.kind == 2) i = dopp<Q>(i);
  return g;
}
// Whether pass op writes population i at cell g.
template <int Q>
__device__ __forceinline__ bool pass_writes(const FaceOp &op, const int *n, const PassCell &g, int i) {
  const int e[3] = {DT<Q>::ex(i), DT<Q>::ey(i), DT<Q>::ez(i)};
  bool w = true;
#pragma unroll
  for (int d = 0; d < (Q == 27 ? 3 : 2); ++d) {
    if (d == op.axis) {
      w = w && g.c[d] == (op.side ? n[d] : -1) && (op.side ? e[d] < 0 : e[d] > 0);
    } else {
      const int t = op.trim && d == (op.axis == 0 ? 1 : 0) ? 1 : 0;
      w = w && g.c[d] >= -1 + t && g.c[d] <= n[d] - t;
    }
  }
  return w;
}

template <int Q, class ST>
__global__ void __launch_bounds__(256) ref_boundary_kernel(const FillArgs a, const FaceOps ops,
                                                           const LinkArgs la) {
  using E = typename Store<ST>::elem;
  asm volatile("griddepcontrol.launch_dependents;");
  if ((int)blockIdx.x < la.blocks) {
    links_block<Q, ST>(la);
    return;
  }
  const Layout &L = a.L;
  const int n[3] = {L.nx, L.ny, L.nz};
  const int t = ((int)blockIdx.x - la.blocks) * 256 + (int)threadIdx.x;
  if (t >= ops.start[ops.n]) return;
  int p = 0;
  while (t >= ops.start[p + 1]) ++p;
  const FaceOp &op = ops.op[p];
  const int ta = op.axis == 0 ? 1 : 0, tb = op.axis == 2 ? 1 : 2;
  const int na = n[ta] + 2, nb = Q == 27 ? n[tb] + 2 : 1;
  const int r = t - ops.start[p], kr = r / (na * nb), rem = r - kr * na * nb;
  int i = (int)((op.dirs >> (5 * (ops.first[p] + kr))) & 31u);
  PassCell g;
  g.c[2] = 0;
  const int pb = rem / na, pa = rem - pb * na - 1;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    if (d == op.axis) g.c[d] = op.side ? n[d] : -1;
    else if (d == ta) g.c[d] = pa;
    else if (Q == 27) g.c[d] = pb - 1;
  }
  if (op.trim && (pa < 0 || pa >= n[ta])) return;  // the ghost ends of the range
  for (int e = p + 1; e < ops.n; ++e)  // edges: the last pass has the last word
    if (pass_writes<Q>(ops.op[e], n, g, i)) return;
  const long long dst = i * L.S + L.idx(g.c[0], g.c[1], g.c[2]);
  int q = p;
  for (;;) {
    g = pass_source<Q>(ops.op[q], n, g, i);
    int e = q - 1;
    while (e >= 0 && !pass_writes<Q>(ops.op[e], n, g, i)) --e;
    if (e < 0) break;
    q = e;
  }
  const long long src = i * L.S + L.idx(g.c[0], g.c[1], g.c[2]);
  const E *from = static_cast<const E *>(L.interior(g.c[0], g.c[1], g.c[2]) ? a.f : a.f2);
  asm volatile("griddepcontrol.wait;" ::: "memory");
  static_cast<E *>(a.f)[dst] = *static_cast<const volatile E *>(from + src);
}

// Ghost layers of A copied into B: once, after the initial fields are written,
// so that both buffers start with the reference's initial ghost values.
template <int Q, class ST>
__global__ void ghost_copy_kernel(const Layout L, const void *src_, void *dst_) {
  using E = typename Store<ST>::elem;
  const E *src = static_cast<const E *>(src_);
  E *dst = static_cast<E *>(dst_);
  const long long cells = (long long)L.px * L.nyp * L.nzp;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < cells;
       t += (long long)gridDim.x * blockDim.x) {
    const int x = (int)(t % L.px) - L.xoff;
    const long long r = t / L.px;
    const int y = (int)(r % L.nyp) - L.G;
    const int z = (int)(r / L.nyp) - L.Gz;
    if (L.interior(x, y, z)) continue;
    const long long e = L.idx(x, y, z);
#pragma unroll 9
    for (int i = 0; i < Q; ++i) dst[i * L.S + e] = src[i * L.S + e];
  }
}

// ---- initialisation ---------------------------------------------------------------
// f = feq(p, u) over the whole ghosted box from host-computed macroscopic fields
// (reference profiles: "3D.../lbm.cpp:245-254", "MPI Kokkos/lbm.cpp:116-124").
template <int Q, class ST>
__global__ void init_macros_kernel(const Layout L, void *f_, const double *u, const double *v,
                                   const double *w, const double *p) {
  using E = typename Store<ST>::elem;
  E *f = static_cast<E *>(f_);
  const int lxp = L.nx + 2 * L.G, lyp = L.ny + 2 * L.G, lzp = L.nz + 2 * L.Gz;
  const long long total = (long long)lxp * lyp * lzp;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x) {
    const int x = (int)(t % lxp) - L.G;
    const int y = (int)((t / lxp) % lyp) - L.G;
    const int z = (int)(t / ((long long)lxp * lyp)) - L.Gz;
    const double uu = u[t], vv = v[t], ww = w[t], pp = p[t];
    const long long c = L.idx(x, y, z);
    for (int i = 0; i < Q; ++i) {
      const double edu = DT<Q>::ex(i) * uu + DT<Q>::ey(i) * vv + DT<Q>::ez(i) * ww;
      const double udu = uu * uu + vv * vv + ww * ww;
      const double feq =
          Lat<Q>::w(i) * pp * 3.0 + Lat<Q>::w(i) * (3.0 * edu + 4.5 * edu * edu - 1.5 * udu);
      f[i * L.S + c] = Dec<ST>::template put<Q>(feq, i, L);
    }
  }
}

// Channel profile: p = 0, u = (u_in, seeded perturbation, 0) in fluid, 0 in
// solids; f = feq.  Also records these as the step-0 macroscopic fields.
template <int Q, class ST>
__global__ void init_channel_kernel(const Layout L, void *f_, const uint32_t *mask, int nxw,
                                    double u_in, double amp, unsigned long long seed,
                                    const float *alpha, double omega,
                                    double *mu, double *mv, double *mw, double *mp) {
  using E = typename Store<ST>::elem;
  E *f = static_cast<E *>(f_);
  const long long total = (long long)L.nx * L.ny * L.nz;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x) {
    const int x = (int)(t % L.nx);
    const int y = (int)((t / L.nx) % L.ny);
    const int z = (int)(t / ((long long)L.nx * L.ny));
    const bool solid = mask_solid(mask, nxw, L.ny, x, y, z);
    const double uu = solid ? 0.0 : u_in;
    const double vv = solid ? 0.0 : perturbation(seed, t, amp);
    mu[t] = uu;
    mv[t] = vv;
    mw[t] = 0.0;
    mp[t] = 0.0;
    const long long c = L.idx(x, y, z);
    // The state is post-collision: the first collision relaxes f = feq(u) toward
    // feq((1 - alpha) u), the identity without porosity.
    const double s = alpha ? 1.0 - (double)alpha[t] : 1.0;
    for (int i = 0; i < Q; ++i) {
      const double edu = DT<Q>::ex(i) * uu + DT<Q>::ey(i) * vv;
      const double udu = uu * uu + vv * vv;
      const double f0 = Lat<Q>::w(i) * 0.0 * 3.0 +
                        Lat<Q>::w(i) * (3.0 * edu + 4.5 * edu * edu - 1.5 * udu);
      double fp = f0;
      if (alpha) {
        const double eb = s * edu, ub = s * s * udu;
        const double fb = Lat<Q>::w(i) * 0.0 * 3.0 +
                          Lat<Q>::w(i) * (3.0 * eb + 4.5 * eb * eb - 1.5 * ub);
        fp = f0 - (f0 - fb) * omega;
      }
      f[i * L.S + c] = Dec<ST>::template put<Q>(fp, i, L);
    }
  }
}

// ---- FP64 domain sums (mass = sum of rho over fluid, momentum) ------------------
// A warp takes 32-cell tiles of rows; per cell the moments are the exact integer
// sums of fixed.cuh (27 slots of the FP64 pipe and 12 for the four sums, against 135
// with FP64 additions per population), per thread and over blocks FP64 sums in a
// fixed order.  256x64x64 FP32: 0.94 -> 0.19 ms (there the last block's one thread had
// also added 4 x 2048 partials one by one).
template <int Q, class ST>
__global__ void __launch_bounds__(256) reduce_mass_kernel(const ReduceArgs a) {
  using LQ = Lat<Q>;
  using E = typename Store<ST>::elem;
  const E *f = static_cast<const E *>(a.f);
  const Layout &L = a.L;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const long long rows = (long long)L.ny * L.nz, tiles = rows * a.nxw;
  const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
  long long fluid = 0;
  for (long long t = blockIdx.x * (long long)(blockDim.x >> 5) + wid; t < tiles; t += warps) {
    const long long row = t / a.nxw;
    const int y = (int)(row % L.ny), z = (int)(row / L.ny);
    const int x = (int)(t - row * a.nxw) * 32 + lane;
    if (x >= L.nx || ((a.mask[t] >> lane) & 1u)) continue;
    const E *p = f + L.idx(x, y, z);
    double v[Q];
    unsigned low = ~0u;  // least nonzero magnitude, twice its bits less 1
    static_for(
        [&](auto ic) {
          constexpr int I = decltype(ic)::value;
          if constexpr (std::is_same<ST, float>::value) {
            v[I] = f2d_bits(p[I * L.S]);
            low = min(low, (__float_as_uint(p[I * L.S]) << 1) - 1u);
          } else {
            v[I] = Dec<ST>::template get<Q>(p[I * L.S], I, L);
          }
        },
        std::make_integer_sequence<int, Q>{});
    if constexpr (std::is_same<ST, float>::value)
      if (low < 0x00FFFFFFu)  // subnormals, which f2d_bits makes zeros (converted at each
                              // load: 637 -> 1,031 us at 512x128x128; with this test 659)
        static_for(
            [&](auto ic) {
              constexpr int I = decltype(ic)::value;
              v[I] = (double)static_cast<const volatile float *>(p)[I * L.S];
            },
            std::make_integer_sequence<int, Q>{});
    ++fluid;
    const int eb = fx_exponent<LQ>(v, 0.0);
    if (eb <= FX_EMAX) {
      long long q[Q], mr, mu[3];
      fx_moments<LQ>(v, eb, q, mr, mu);
      const double su = __hiloint2double((eb - FX_P - Fx<LQ>::U) << 20, 0);
      const double sr = __hiloint2double((eb - FX_P - Fx<LQ>::R) << 20, 0);
      acc[0] = __fma_rn(__ll2double_rn(mr), sr, acc[0]);
#pragma unroll
      for (int d = 0; d < 3; ++d) acc[1 + d] = __fma_rn(__ll2double_rn(mu[d]), su, acc[1 + d]);
    } else {
      static_for(
          [&](auto ic) {
            constexpr int I = decltype(ic)::value;
            acc[0] += v[I];
            acc[1] += v[I] * LQ::ex(I);
            acc[2] += v[I] * LQ::ey(I);
            acc[3] += v[I] * LQ::ez(I);
          },
          std::make_integer_sequence<int, Q>{});
    }
  }
  acc[0] += (double)fluid;  // rho = 1 + sum f
  __shared__ double sh[4][32];
  __shared__ bool last;
  auto block_sums = [&] {  // valid in thread 0
    for (int o = 16; o > 0; o >>= 1)
      for (int q = 0; q < 4; ++q) acc[q] += __shfl_down_sync(0xffffffffu, acc[q], o);
    if (lane == 0)
      for (int q = 0; q < 4; ++q) sh[q][wid] = acc[q];
    __syncthreads();
    if (threadIdx.x == 0)
      for (int q = 0; q < 4; ++q) {
        acc[q] = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) acc[q] += sh[q][w];
      }
  };
  block_sums();
  if (threadIdx.x == 0) {
    for (int q = 0; q < 4; ++q) a.partials[4 * blockIdx.x + q] = acc[q];
    __threadfence();
    last = (atomicAdd(a.counter, 1u) == gridDim.x - 1);
  }
  __syncthreads();
  if (last) {
    __threadfence();
    const volatile double *p = a.partials;
    for (int q = 0; q < 4; ++q) acc[q] = 0.0;
    for (unsigned b = threadIdx.x; b < gridDim.x; b += blockDim.x)
      for (int q = 0; q < 4; ++q) acc[q] += p[4 * b + q];
    __syncthreads();
    block_sums();
    if (threadIdx.x == 0) {
      for (int q = 0; q < 4; ++q) a.out[q] = acc[q];
      *a.counter = 0u;
    }
  }
}

// ---- dump / restore --------------------------------------------------------------
// Rows [r0, r0 + n) of the dense [i][z][y][x] state, one warp per row, to or from
// `dense` (row r0 first).
template <int Q, class ST, bool PUT>
__global__ void __launch_bounds__(256) dense_rows_kernel(const Layout L, void *f_, double *dense,
                                                         long long r0, long long n) {
  using E = typename Store<ST>::elem;
  E *f = static_cast<E *>(f_);
  const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
  for (long long k = blockIdx.x * (long long)(blockDim.x >> 5) + (threadIdx.x >> 5); k < n;
       k += warps) {
    const long long r = r0 + k, yz = r % ((long long)L.ny * L.nz);
    const int i = (int)(r / ((long long)L.ny * L.nz));
    E *p = f + i * L.S + L.idx(0, (int)(yz % L.ny), (int)(yz / L.ny));
    double *d = dense + k * L.nx;
    for (int x = threadIdx.x & 31; x < L.nx; x += 32) {
      if constexpr (PUT) p[x] = Dec<ST>::template put<Q>(d[x], i, L);
      else d[x] = Dec<ST>::template get<Q>(p[x], i, L);
    }
  }
}

}  // namespace

long long launches() { return __atomic_load_n(&g_launches, __ATOMIC_RELAXED); }
void count_launch(long long n) { __atomic_fetch_add(&g_launches, n, __ATOMIC_RELAXED); }

cudaError_t launch_sweep_q9(int store, int compute, const SweepArgs &a, cudaStream_t s);
cudaError_t launch_sweep_q27(int store, int compute, const SweepArgs &a, cudaStream_t s);

cudaError_t launch_sweep(int Q, int store, int compute, const SweepArgs &a, cudaStream_t s) {
  return Q == 9 ? launch_sweep_q9(store, compute, a, s) : launch_sweep_q27(store, compute, a, s);
}

cudaError_t launch_sweep_channel_q9(int store, int compute, const SweepArgs &a, cudaStream_t s);
cudaError_t launch_sweep_channel_q27(int store, int compute, const SweepArgs &a, cudaStream_t s);

cudaError_t launch_macros_channel_q9(int store, int compute, const SweepArgs &a, cudaStream_t s);
cudaError_t launch_macros_channel_q27(int store, int compute, const SweepArgs &a,
                                      cudaStream_t s);

cudaError_t launch_macros_channel(int Q, int store, int compute, const SweepArgs &a,
                                  cudaStream_t s) {
  return Q == 9 ? launch_macros_channel_q9(store, compute, a, s)
                : launch_macros_channel_q27(store, compute, a, s);
}

cudaError_t launch_stream_state_q9(int store, const SweepArgs &a, bool ref, double *out,
                                   cudaStream_t s);
cudaError_t launch_stream_state_q27(int store, const SweepArgs &a, bool ref, double *out,
                                    cudaStream_t s);
cudaError_t launch_stream_state(int Q, int store, const SweepArgs &a, bool ref, double *out,
                                cudaStream_t s) {
  return Q == 9 ? launch_stream_state_q9(store, a, ref, out, s)
                : launch_stream_state_q27(store, a, ref, out, s);
}

cudaError_t launch_sweep_channel(int Q, int store, int compute, const SweepArgs &a,
                                 cudaStream_t s) {
  return Q == 9 ? launch_sweep_channel_q9(store, compute, a, s)
                : launch_sweep_channel_q27(store, compute, a, s);
}

// Dispatch helper: run F<Q, ST> for the runtime (Q, store).
#define CFLBM_DISPATCH(Q, store, CALL)                                   \
  do {                                                                   \
    if ((Q) == 9) {                                                      \
      constexpr int QQ = 9;                                              \
      if ((store) == STORE_F64) { using ST = double; CALL; }             \
      else if ((store) == STORE_F32) { using ST = float; CALL; }         \
      else { using ST = F16Dev; CALL; }                                  \
    } else {                                                             \
      constexpr int QQ = 27;                                             \
      if ((store) == STORE_F64) { using ST = double; CALL; }             \
      else if ((store) == STORE_F32) { using ST = float; CALL; }         \
      else { using ST = F16Dev; CALL; }                                  \
    }                                                                    \
  } while (0)

// The populations a pass writes: e along its axis positive (inlet copy, low wall)
// or negative (outlet extrapolation, high wall) -- 9 in D3Q27, 3 in D2Q9.
static void face_dirs(int Q, FaceOp &op) {
  op.ndir = 0;
  op.dirs = 0;
  for (int i = 1; i < Q; ++i) {
    const int e[3] = {Q == 27 ? Lat<27>::ex(i) : Lat<9>::ex(i),
                      Q == 27 ? Lat<27>::ey(i) : Lat<9>::ey(i),
                      Q == 27 ? Lat<27>::ez(i) : 0};
    const int ea = e[op.axis];
    const bool want = op.kind == 0 ? ea > 0 : (op.kind == 1 ? ea < 0 : (op.side == 0 ? ea > 0 : ea < 0));
    if (want && op.ndir < 9) op.dirs |= (unsigned long long)i << (5 * op.ndir++);
  }
}

cudaError_t launch_ref_boundary(int Q, int store, const FillArgs &a, const FaceOp *op, int nops,
                                const LinkArgs &la0, cudaStream_t s) {
  LinkArgs la = la0;
  FaceOps ops{};
  ops.n = nops;
  const int n[3] = {a.L.nx, a.L.ny, a.L.nz};
  long long cells[6] = {};
  for (int p = 0; p < nops; ++p) {
    ops.op[p] = op[p];
    face_dirs(Q, ops.op[p]);
    const int ta = op[p].axis == 0 ? 1 : 0, tb = op[p].axis == 2 ? 1 : 2;
    cells[p] = (long long)(n[ta] + 2) * (Q == 27 ? n[tb] + 2 : 1);
  }
  int p = 0, k = 0;
  do {
    if (!next_faces(ops, cells, FACE_THREADS, p, k)) return cudaErrorInvalidValue;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(la.blocks + (ops.start[nops] + 255) / 256));
    cfg.blockDim = dim3(256);
    cfg.stream = s;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    cudaError_t e = cudaSuccess;
    CFLBM_DISPATCH(Q, store,
                   (e = cudaLaunchKernelEx(&cfg, ref_boundary_kernel<QQ, ST>, a, ops, la)));
    if (e != cudaSuccess) return e;
    count_launch();
    la.blocks = 0;  // the links go with the first
  } while (p < nops);
  return cudaGetLastError();
}

cudaError_t launch_ghost_copy(int Q, int store, const Layout &L, const void *src, void *dst,
                              cudaStream_t s) {
  const int blocks = blocks_for((long long)L.px * L.nyp * L.nzp, 256);
  CFLBM_DISPATCH(Q, store, (ghost_copy_kernel<QQ, ST><<<blocks, 256, 0, s>>>(L, src, dst)));
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_init_macros(int Q, int store, const Layout &L, void *f, const double *u,
                               const double *v, const double *w, const double *p,
                               cudaStream_t s) {
  const long long total =
      (long long)(L.nx + 2 * L.G) * (L.ny + 2 * L.G) * (L.nz + 2 * L.Gz);
  const int blocks = blocks_for(total, 256);
  CFLBM_DISPATCH(Q, store,
                 (init_macros_kernel<QQ, ST><<<blocks, 256, 0, s>>>(L, f, u, v, w, p)));
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_init_channel(int Q, int store, const Layout &L, void *f,
                                const uint32_t *mask, int nxw, double u_in, double amp,
                                unsigned long long seed, const float *alpha, double omega,
                                double *mu, double *mv, double *mw, double *mp, cudaStream_t s) {
  const int blocks = blocks_for((long long)L.nx * L.ny * L.nz, 256);
  CFLBM_DISPATCH(Q, store,
                 (init_channel_kernel<QQ, ST><<<blocks, 256, 0, s>>>(
                     L, f, mask, nxw, u_in, amp, seed, alpha, omega, mu, mv, mw, mp)));
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_reduce_mass(int Q, int store, const ReduceArgs &a, int blocks,
                               cudaStream_t s) {
  CFLBM_DISPATCH(Q, store, (reduce_mass_kernel<QQ, ST><<<blocks, 256, 0, s>>>(a)));
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_dense_rows(int Q, int store, const Layout &L, void *f, double *dense,
                              long long r0, long long n, bool put, cudaStream_t s) {
  const int blocks = blocks_for((n + 7) / 8, 1);
  if (put)
    CFLBM_DISPATCH(Q, store, (dense_rows_kernel<QQ, ST, true><<<blocks, 256, 0, s>>>(L, f, dense, r0, n)));
  else
    CFLBM_DISPATCH(Q, store, (dense_rows_kernel<QQ, ST, false><<<blocks, 256, 0, s>>>(L, f, dense, r0, n)));
  count_launch();
  return cudaGetLastError();
}

}  // namespace cflbm

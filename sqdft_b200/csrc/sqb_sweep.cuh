#pragma once
// Sweep kernel: the per-grid-node work of the SQ step (Lanczos bounds and
// Chebyshev moments, ClenshawCurtisSpectralQuadrature sq.cpp:530-661) on
// sm_100a, built around a branch-free nonlocal term.
//
// Persistent CTAs, as many as fit on an SM, take grid nodes from an atomic queue.  Every
// matvec H v = -1/2 Lap_h v + Veff v + Vnl v on a node's (2nloc+1)^3 window
// (HsubTimesVec sq.cpp:838-929, VnlocsubTimesVec nonlocal.cpp:20-215; v zero
// outside the window) is one sweep over the window's z-planes:
//   * each thread owns a pair of window columns x and RY adjacent rows y; it
//     writes its centre values into a shared-memory plane with a zero halo of
//     6, so the x and y neighbours are unconditional loads (the window
//     truncation falls out of the halo); the pair shares its x-arm loads (16
//     bytes each) and the RY rows their y-arm loads;
//   * the 2 FDN + 1 planes of a column's stencil: the centre and the FDN
//     planes ahead in registers, the FDN planes behind in the thread's own
//     slots of a shared ring (no barrier: no other thread reads them);
//   * the shared planes rotate through three buffers under a split barrier:
//     a warp writes plane z + 1 and arrives on an mbarrier before it works
//     on plane z, and waits for that phase (bounded) only afterwards, so
//     warps drift by up to a plane instead of meeting at every plane;
//   * the nonlocal term reads the layered projector fields (sqb_internal.cuh):
//     per point and layer one 16-bit projector base and the projector values,
//     so the gather sum_J c_J chi_J(x) is a fixed loop over four layers with
//     no per-box control flow, c_J read from a shared array indexed by the
//     global projector id;
//   * the dot products chi_J . w of the sweep's output w, which the next
//     matvec needs, are accumulated per thread along z for each layer; when a
//     column leaves a ball (the layer's id changes) the column's partial sum
//     goes to the CTA's flush buffer in global memory, at the slot of (layer,
//     the ball's last window plane, column), which no other ball shares; after
//     the last plane every warp sums whole balls from it in a fixed order:
//     deterministic, one reduction per ball per sweep, none inside the plane
//     loop.
// Lanczos keeps the reference's recurrence, start vector and convergence test
// (sq.cpp:965-1092) with one sweep per step: the sweep forms the next
// unnormalised Lanczos vector from the stored vectors while loading it, and
// the block then finds the extreme eigenvalues of the tridiagonal (the
// quantities TridiagEigenSolve sq.cpp:1094-1180 returns) by a
// (16 warps + 1)-way multisection (33-way on two warps, 481-way on thirty).  Chebyshev moments use the reference's doubling identities
// (sq.cpp:564-655).  The Lanczos-quadrature form takes bounds and moments from
// one Lanczos run started at the node (Gauss-quadrature identity).
#include <cmath>
#include <cstdio>
#include <type_traits>

#include "sqb_internal.cuh"

namespace sqb {
namespace sweep {

constexpr int KL = LAYERS;

// Sweep kinds: the Lanczos start vector's projections only; a Lanczos step;
// a Chebyshev step; a Chebyshev step that also accumulates the density-matrix
// column D += c t_k+1 / h^3 (ForcesNonLocal).
enum : int { SK_ONES = 0, SK_LZF = 1, SK_CH = 2, SK_FD = 3 };

struct Shared {
  unsigned long long pbar;  // plane barrier of the sweeps (mbarrier, one arrival per warp and plane)
  unsigned pbar_phase;      // its phases completed so far
  int wabort;               // a plane wait ran out of time: later waits are skipped
  int node, qidx, gi, gj, gk;
  int n_ent, n_pi;
  int stop, count;
  double center_val;
  double scal[2];
  double red[32][2];
  double red3[32][3];
  double scal2[3];
  double aa[MAXL];
  double bb[MAXL];
  double b2[MAXL];  // bb^2
  double ger[2];    // Gershgorin interval of the rows whose both neighbours are known
  double eig[2], eprev[2];
  double wdel[2];   // last changes of the extremes (warm start of the next multisection)
  int warm;         // eig holds the extremes of the previous, one row smaller tridiagonal
  double br[2][2];  // multisection brackets (lambda_min, lambda_max)
  int wres[32];     // per-warp multisection results
  int scan[33];
  // boxes (replica balls meeting the window), window coordinates
  short e_x0[MAXE], e_x1[MAXE], e_y0[MAXE], e_y1[MAXE], e_z0[MAXE], e_z1[MAXE];
  unsigned char e_k[MAXE], e_np[MAXE], e_t[MAXE];
  short e_pb[MAXE];  // first local projector instance
  int e_gpb[MAXE];   // first global projector id
  int e_atom[MAXE];  // global atom (force passes)
  int e_r[MAXE];     // index of the replica's box
  // local projector instances p < n_pi
  short pi_e[MAXP];
  int pi_g[MAXP];
  double p_nxt[MAXP];  // chi^T w of the sweep's output
  double p_in[MAXP];   // chi^T W of a Lanczos sweep's input (one projector per layer slot)
  double p_den[MAXP];
  double pw_cur[MAXP];   // Lanczos: chi^T W_m
  double pw_prev[MAXP];  // Lanczos: chi^T W_m-1
};

// Thread tile: a pair of adjacent window columns (one 16-byte shared or global
// access in FP64) and RY adjacent rows.  The pairs start at even columns of the
// extended grid, so a window that starts at an odd column is shifted by one
// (sh = gi & 1): window column x sits at pair column x + sh of 0 .. n, and one
// pad column per row (x = -1 or x = n) carries zeros.  Window vectors, plane
// buffers and flush slots use this pair layout, rows of pair_cols(n) values.
__host__ __device__ constexpr int pair_cols(int n) { return n + 1; }  // n is odd
__host__ __device__ constexpr size_t vec_points(int n) { return (size_t)n * n * pair_cols(n); }
// Plane buffer pitch: the row with its halo, even (16-byte rows), and where
// that is possible = the pairs per row modulo 8, so that eight lanes that run
// over a row's end into the next row of tiles still touch distinct banks.
__host__ __device__ constexpr int plane_pitch(int n) {
  const int hx = pair_cols(n) / 2, p = pair_cols(n) + 2 * FDN;
  return hx % 2 ? p : p + ((hx - p) % 8 + 8) % 8;
}
__host__ __device__ constexpr int plane_rows(int n, int ry) { return n + 2 * FDN + ry - 1; }
// Halo'd planes of the stencil input: plane z lives in buffer z mod NPLANE.
// Three buffers let a thread write plane z + 1 before it works on plane z
// while the slowest thread may still read plane z - 1 (see sweep).
constexpr int NPLANE = 3;
__host__ __device__ inline size_t planes_bytes(int n, int ry) {
  return ((size_t)NPLANE * plane_pitch(n) * plane_rows(n, ry) * sizeof(double) + 127) & ~size_t(127);
}
// Lanczos sweeps of the one-projector fields also accumulate the dot products
// of their input (the exact chi^T W_m, see lanczos), flushed into a second
// set of the flush buffer.  The buffer (per CTA, after the three window
// vectors in the scratch) holds [set][layer][projector][plane][row][pair column].
__host__ __device__ constexpr bool input_dots(int pm) { return pm == 1; }
__host__ __device__ inline size_t flush_doubles(int n, int pm) {
  return (size_t)(input_dots(pm) ? 2 : 1) * KL * pm * vec_points(n);
}
__host__ __device__ inline size_t shared_fixed() { return (sizeof(Shared) + 127) & ~size_t(127); }
// The threads' rings of the FDN planes behind: a plane's slot is free once the
// step FDN planes later has read it, which is the step that refills it.  The
// slots are a compile-time stride (the tile's launch bound) apart.
constexpr int RSLOT = FDN;
__host__ __device__ constexpr size_t ring_bytes(int maxt, int ry) {
  return (size_t)RSLOT * ry * maxt * 2 * sizeof(double);
}
__host__ __device__ inline int sweep_threads_of(int n, int ry) {
  const int t = (pair_cols(n) / 2 * ((n + ry - 1) / ry) + 31) / 32 * 32;
  return t < 64 ? 64 : t;  // two warps at least: the multisection's two extremes
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Barrier of the block's threads inside a sweep (named barrier 1).
__device__ __forceinline__ void bar_sweep(int nthreads) {
  asm volatile("bar.sync 1, %0;\n" ::"r"(nthreads) : "memory");
}

// The plane barrier: an mbarrier in shared memory that every warp of the block
// arrives on once per plane, after a __syncwarp (release: the warp's plane
// writes are visible to the threads whose wait on that phase returns, acquire).
__device__ __forceinline__ unsigned pbar_addr(const unsigned long long *bar) {
  return (unsigned)__cvta_generic_to_shared(bar);
}
__device__ __forceinline__ void pbar_init(unsigned long long *bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(pbar_addr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void pbar_arrive(unsigned long long *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(pbar_addr(bar)) : "memory");
}
__device__ __forceinline__ bool pbar_try_wait(unsigned long long *bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(pbar_addr(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ unsigned long long gtimer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
// Every warp of the block arrives once per plane, so a phase completes in
// microseconds; a wait that outlasts PBAR_WAIT_NS means a warp stopped
// arriving: the wait sets the status bit and the block's abort flag, after
// which no plane wait blocks (the step's results are then void and the call
// returns an error).
constexpr unsigned long long PBAR_WAIT_NS = 2000000000ull;
__device__ __forceinline__ void pbar_wait(Shared &S, int *status, unsigned phase) {
  const unsigned parity = phase & 1u;
  if (pbar_try_wait(&S.pbar, parity)) return;
  const unsigned long long t0 = gtimer_ns();
  while (!pbar_try_wait(&S.pbar, parity)) {
    if (*(volatile int *)&S.wabort) return;
    if (gtimer_ns() - t0 > PBAR_WAIT_NS) {
      *(volatile int *)&S.wabort = 1;
      atomicOr(status, ST_WAIT_LIMIT);
      return;
    }
  }
}
// Set up the plane barrier at the start of a kernel (before any sweep).
__device__ __forceinline__ void pbar_setup(Shared &S) {
  if (threadIdx.x == 0) {
    pbar_init(&S.pbar, blockDim.x / 32);
    S.pbar_phase = 0u;
    S.wabort = 0;
  }
  __syncthreads();
}

template <typename T>
struct IO {
  const T *vin = nullptr;  // stencil input (LZF: Y = H W_m-1; CH: t_k)
  T *out = nullptr;        // output (LZF: H W_m; CH: t_k+1)
  const T *p1 = nullptr;   // LZF: W_m-1; CH: t_k-1
  const T *p2 = nullptr;   // LZF: W_m-2
  T *wout = nullptr;       // LZF: where the formed W_m is stored
  double s1 = 1.0;         // LZF: W_m = s1 (Y - ca W1) - cb W2
  double ca = 0.0, cb = 0.0;  // LZF: a, b s; CH: chi, zee
  double chk = 0.0;        // ONES: start vector 1 + chk (-1)^(x+y+z)
  int first = 0;           // CH: t_1 = (H t_0 - chi t_0) / zee (no t_k-1 term)
  int dbl = 0;             // CH: accumulate <t_k+1, t_k+1> and <t_k+1, t_k> (doubling)
  double *dacc = nullptr;  // FD: density-matrix column, FP64
  double cd = 0.0, ce = 0.0;  // FD: D += t_k+1 cd / h^3 (first: D = e_c ce / h^3 + t_1 cd / h^3)
};

// Lanczos start vector at window index g: 1 + chk (-1)^(x+y+z); the window
// edge n is odd, so x + y + z and g = (z n + y) n + x have the same parity, and
// any g of that parity will do.
__device__ __forceinline__ double start_val(double chk, int g) { return 1.0 + chk * (1.0 - 2.0 * (double)(g & 1)); }

__device__ __forceinline__ unsigned lay_of(unsigned long long w, int k) {
  return (unsigned)(w >> (16 * k)) & 0xffffu;
}

template <typename T>
__device__ __forceinline__ T *slot(const SweepArgs &a, int k) {
  return reinterpret_cast<T *>(a.scratch + blockIdx.x * a.scratch_stride + (size_t)k * vec_points(a.n) * sizeof(double));
}

// Sums of the flushed column partials of every projector instance over its
// box's columns, at the slots of its ball's last window plane, into p_nxt;
// with IND also the input dots of the second set, into p_in.  Eight lanes per
// instance in a fixed order, four instances per warp at a time, eight loads
// in flight per lane: the loads' latency is what this costs.
template <int PM, bool IND>
__device__ __forceinline__ void reduce_instances(const SweepArgs &a, Shared &S, const double *fb, int warp, int nwarp,
                                                 int lane) {
  const int n = a.n, NP = pair_cols(n), plane = n * NP, set = KL * PM * n * plane;
  const int sh = S.gi & 1, sub = lane & 7;
  for (int p0 = warp * 4; p0 < S.n_pi; p0 += nwarp * 4) {
    const int p = p0 + (lane >> 3);
    double s = 0.0, sw = 0.0;
    if (p < S.n_pi) {
      const int e = S.pi_e[p], q = p - S.e_pb[e], k = S.e_k[e];
      const int x0 = S.e_x0[e], y0 = S.e_y0[e];
      const int bx = S.e_x1[e] - x0 + 1, cnt = bx * (S.e_y1[e] - y0 + 1);
      const int base = ((k * PM + q) * n + S.e_z1[e]) * plane + y0 * NP + x0 + sh;
      // i / bx for i < 43 * 43 by a 2^20 reciprocal: the excess i (inv bx - 2^20) / (bx 2^20) stays below 1 / bx
      const unsigned inv = ((1u << 20) + bx - 1) / bx;
      const double *f = fb + base;
      for (int i0 = sub; i0 < cnt; i0 += 64) {
        double v[8], w[8];
#pragma unroll
        for (int t = 0; t < 8; t++) {
          const int i = i0 + 8 * t, yy = (int)(((unsigned)i * inv) >> 20);
          const bool in = i < cnt;
          const int o = in ? SQB_IDX(base + yy * NP + (i - yy * bx), set, a.status) - base : 0;
          v[t] = in ? f[o] : 0.0;
          if constexpr (IND) w[t] = in ? f[o + set] : 0.0;
        }
#pragma unroll
        for (int t = 0; t < 8; t++) {
          s += v[t];
          if constexpr (IND) sw += w[t];
        }
      }
    }
    __syncwarp();
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
      s += __shfl_xor_sync(0xffffffffu, s, o);
      if constexpr (IND) sw += __shfl_xor_sync(0xffffffffu, sw, o);
    }
    if (sub == 0 && p < S.n_pi) {
      S.p_nxt[p] = s;
      if constexpr (IND) S.p_in[p] = sw;
    }
  }
}

// All plane buffers to zero (the halo; the sweeps write the interior).  Once
// per kernel, and where the buffers change between FP32 and FP64 values.
static __device__ void zero_planes(const SweepArgs &a, unsigned char *dyn, int ry) {
  __syncthreads();
  uint4 *p = reinterpret_cast<uint4 *>(dyn);
  for (int i = threadIdx.x; i < (int)(planes_bytes(a.n, ry) / 16); i += blockDim.x) p[i] = make_uint4(0, 0, 0, 0);
  __syncthreads();
}

template <typename T>
struct PairOf;
template <>
struct PairOf<double> {
  using type = double2;
};
template <>
struct PairOf<float> {
  using type = float2;
};

// One sweep over the window's z-planes (all threads of the block).  A
// thread's stencil input along z: the centre and the FDN planes ahead in
// registers (fut[j][0] the centre, fut[j][s] plane z + s) and the FDN planes
// behind in the thread's own slots of a shared ring.
//
// What bounds it is latency and instruction issue (B200, 31^3 windows, force
// sweeps: 49% of issue slots; 298 thread instructions per point, 56 of them
// FP64), not FP64 (17.5% of the pipe) and not memory (132 bytes per point
// through L2, 37 of them to or from DRAM: 2.0 TB/s).  A pair of columns
// per thread takes its x-arm values in 3 16-byte loads per point where a single
// column takes 12 8-byte ones.  The streamed operands bypass L1 (__ldcg,
// __stcg), which the shared memory leaves small, so that it keeps the spilled
// registers: with them in it 60% of the spill loads went to L2.
template <typename T, int PM, int SK, int RY, int NT>
__device__ __forceinline__ void sweep(const SweepArgs &a, Shared &S, unsigned char *dyn, const IO<T> &io,
                                      double &acc0, double &acc1) {
  using T2 = typename PairOf<T>::type;
  constexpr bool STENCIL = SK != SK_ONES;
  constexpr bool CHEB = SK == SK_CH || SK == SK_FD;
  constexpr int F = FDN + 1;       // planes held in registers
  constexpr bool CHR = PM == 1;    // projector values kept in registers from one plane to the next
  constexpr bool IND = SK == SK_LZF && input_dots(PM);  // dot products of the input too
  const int n = a.n, NP = pair_cols(n), HX = NP >> 1, P = plane_pitch(n), PB = P * plane_rows(n, RY);
  const int tid = threadIdx.x, NS = a.nsweep, lane = tid & 31, warp = tid >> 5, nwarp = NS >> 5;
  const int tg = tid / HX, px = tid - tg * HX;
  const bool tv = tg * RY < n;
  const int sh = S.gi & 1;
  const int xx = 2 * px, yb = tv ? tg * RY : 0;  // pair column, first row
  const bool cv0 = !(sh && px == 0), cv1 = sh || px != HX - 1;  // columns inside the window
  const int nl = a.nloc;
  const int EP = a.ex * a.ey, EV = (int)a.evol;  // the extended grid fits 32-bit indices
  const int VP = n * NP, NW = n * VP;            // values per plane and per window vector
  const unsigned dummy = (unsigned)a.n_gproj;
  const unsigned long long empty = 0x0001000100010001ull * (unsigned long long)dummy;  // no ball in any layer
  T *sm = reinterpret_cast<T *>(dyn);
  T2 *ring = reinterpret_cast<T2 *>(dyn + planes_bytes(n, RY)) + tid;
  constexpr int RS = RY * NT;  // pairs per ring slot
  const double *pcur = reinterpret_cast<const double *>(dyn + planes_bytes(n, RY) + ring_bytes(NT, RY));
  double *fb = slot<double>(a, 3);  // flush buffer: [set][layer][projector][plane][row][pair column]
  const int fset = KL * PM * NW;
  int *const st = a.status;  // (bounds-check build)
  (void)st;
  (void)EV;

  bool ok[RY];
#pragma unroll
  for (int j = 0; j < RY; j++) ok[j] = tv && yb + j < n;
  const int g0 = yb * NP + xx;                                                       // window vectors, plane 0
  const int X0 = (S.gk * a.ey + S.gj + yb) * a.ex + S.gi - sh + xx;                  // fields, plane 0
  // the thread that owns the window centre: row cj of its tile, column cc of its pair
  const bool ctr = tv && xx == ((nl + sh) & ~1) && yb <= nl && nl < yb + RY;
  const int cj = nl - yb, cc = (nl + sh) & 1;
  const unsigned par0 = (unsigned)(xx - sh + yb) & 1u;  // parity of x + y of the tile's first point

  // the stencil input of row j at plane zz (LZF: formed from the loaded operands)
  T2 fut[RY][F];
  T2 pf[RY], r1[RY], r2[RY];
  auto load_ops = [&](int j, int zz) {
    if (!ok[j] || zz >= n) return;
    const int g = SQB_IDX(g0 + zz * VP + j * NP, NW - 1, st);
    pf[j] = __ldcg(reinterpret_cast<const T2 *>(io.vin + g));
    if constexpr (SK == SK_LZF) {
      r1[j] = __ldcg(reinterpret_cast<const T2 *>(io.p1 + g));
      r2[j] = __ldcg(reinterpret_cast<const T2 *>(io.p2 + g));
    }
  };
  auto next_in = [&](int j, int zz) -> T2 {
    T2 v;
    v.x = v.y = T(0);
    if (!ok[j] || zz >= n) return v;
    if constexpr (SK == SK_LZF) {
      v.x = (T)(io.s1 * ((double)pf[j].x - io.ca * (double)r1[j].x) - io.cb * (double)r2[j].x);
      v.y = (T)(io.s1 * ((double)pf[j].y - io.ca * (double)r1[j].y) - io.cb * (double)r2[j].y);
    } else {
      v = pf[j];
    }
    if constexpr (SK == SK_LZF)
      __stcg(reinterpret_cast<T2 *>(io.wout + SQB_IDX(g0 + zz * VP + j * NP, NW - 1, st)), v);
    return v;
  };

  // per-plane point data, loaded one plane ahead
  double2 ve[RY];
  T2 q1[RY];
  double2 dq[RY];  // FD: D at the point
  unsigned long long idc[RY][2] = {}, idn[RY][2] = {};
  double2 chc[RY][KL];       // CHR: projector values
  double2 acd[RY][KL][PM];   // dot products with the output, per column and current ball
  double2 acw[RY][KL];       // IND: with the input
  auto load_ids = [&](int j, int zz) {
    ulonglong2 v = make_ulonglong2(empty, empty);
    if (ok[j] && zz < n)
      v = __ldcg(reinterpret_cast<const ulonglong2 *>(a.lay_id + SQB_IDX(X0 + zz * EP + j * a.ex, EV - 1, st)));
    idn[j][0] = v.x;
    idn[j][1] = v.y;
  };
  auto chi_ld = [&](int j, int kq, int k, int X) -> double2 {
    double2 v = make_double2(0.0, 0.0);
    if (lay_of(idc[j][0], k) != dummy || lay_of(idc[j][1], k) != dummy)
      v = CHR ? __ldcg(reinterpret_cast<const double2 *>(a.lay_chi + (size_t)kq * EV + X))
              : __ldg(reinterpret_cast<const double2 *>(a.lay_chi + (size_t)kq * EV + X));
    return v;
  };
  auto load_point = [&](int j, int zz) {
    if (!ok[j] || zz >= n) return;
    const int X = SQB_IDX(X0 + zz * EP + j * a.ex, EV - 1, st);
    if constexpr (STENCIL) ve[j] = __ldcg(reinterpret_cast<const double2 *>(a.veff64 + X));
    if constexpr (CHEB) {
      if (!io.first) {
        q1[j] = __ldcg(reinterpret_cast<const T2 *>(io.p1 + SQB_IDX(g0 + zz * VP + j * NP, NW - 1, st)));
      }
    }
    if constexpr (SK == SK_FD) {
      if (!io.first) dq[j] = __ldcg(reinterpret_cast<const double2 *>(io.dacc + SQB_IDX(g0 + zz * VP + j * NP, NW - 1, st)));
    }
    if constexpr (CHR) {
#pragma unroll
      for (int k = 0; k < KL; k++) chc[j][k] = chi_ld(j, k, k, X);
    }
  };

#pragma unroll
  for (int j = 0; j < RY; j++) {
    ve[j] = dq[j] = make_double2(0.0, 0.0);
    q1[j].x = q1[j].y = T(0);
    load_ids(j, 0);
#pragma unroll
    for (int i = 0; i < 2; i++) idc[j][i] = idn[j][i];
#pragma unroll
    for (int k = 0; k < KL; k++) {
      acw[j][k] = chc[j][k] = make_double2(0.0, 0.0);
#pragma unroll
      for (int q = 0; q < PM; q++) acd[j][k][q] = make_double2(0.0, 0.0);
    }
    load_ids(j, 1);
    if constexpr (STENCIL) {
      // planes behind the window are zero; planes 0..FDN enter it
      T2 zero;
      zero.x = zero.y = T(0);
#pragma unroll
      for (int s = 0; s < RSLOT; s++) ring[s * RS + j * NT] = zero;
      T2 pp[FDN + 1], pr1[FDN + 1], pr2[FDN + 1];  // (all loads in flight before the first stored plane)
#pragma unroll
      for (int s = 0; s <= FDN; s++) {
        load_ops(j, s);
        pp[s] = pf[j];
        if constexpr (SK == SK_LZF) {
          pr1[s] = r1[j];
          pr2[s] = r2[j];
        }
      }
#pragma unroll
      for (int s = 0; s <= FDN; s++) {
        pf[j] = pp[s];
        if constexpr (SK == SK_LZF) {
          r1[j] = pr1[s];
          r2[j] = pr2[s];
        }
        fut[j][s] = next_in(j, s);
      }
      load_ops(j, FDN + 1);
    }
    load_point(j, 0);
  }
  const double c0 = 3.0 * a.coeff_lap[0];
  const double rcb = CHEB ? (io.first ? 1.0 : 2.0) / io.cb : 0.0;  // (2/zee is exactly twice 1/zee)
  const double cdh = io.cd / a.h3, ceh = io.ce / a.h3;
  unsigned big = 0u;  // largest magnitude word of the outputs (non-finite check)

  // Planes through the shared buffers with a split barrier: in step z a
  // thread first writes its centre values of plane z + 1 (buffer (z+1) mod 3)
  // and its warp arrives, then works on plane z, and only then waits until
  // every warp has written plane z + 1.  A warp in step z has seen every warp
  // arrive in step z - 1, so the slowest is at worst in step z - 1, reading
  // buffer (z-1) mod 3: one buffer apart from the one written.  Warps drift
  // by up to a plane instead of meeting at every plane.
  const int sofs = (yb + FDN) * P + xx + FDN;  // the thread's first row in a plane buffer
  if constexpr (STENCIL) {
    if (tv) {
#pragma unroll
      for (int j = 0; j < RY; j++) *reinterpret_cast<T2 *>(sm + sofs + j * P) = fut[j][0];
    }
  }
  bar_sweep(NS);  // plane 0 written; the previous sweep's phases are counted
  const unsigned ph0 = S.pbar_phase;
  int bz = 0;  // buffer of plane z
  int rz = 0;  // ring slot of plane z (and of plane z - RSLOT)
  for (int z = 0; z < n; z++) {
    const T *smz = sm + bz * PB;
    const int bn = bz == NPLANE - 1 ? 0 : bz + 1;
    if constexpr (STENCIL) {
      if (z + 1 < n) {
        if (tv) {
#pragma unroll
          for (int j = 0; j < RY; j++) *reinterpret_cast<T2 *>(sm + bn * PB + sofs + j * P) = fut[j][1];
        }
        __syncwarp();
        if (lane == 0) pbar_arrive(&S.pbar);
      }
    }
    if (tv) {
      double2 hv[RY], v[RY];
      if constexpr (STENCIL) {
        // arm k of each point sums (x-k) + (x+k) + (y-k) + (y+k) + (z-k) + (z+k)
        // in that order before the coefficient, as HsubTimesVec does
        // (sq.cpp:894-897).  The RY rows y0..y0+RY-1 of a thread share their
        // y-arm loads: arm k loads rows y0-k (ym[k]) and y0+RY-1+k (yp[k]); row
        // j's y0+j-k is the centre of row j-k when j >= k, else ym[k-j], and
        // its y0+j+k the centre of row j+k when j+k < RY, else yp[j+k-RY+1].
        const T *cp = smz + sofs;
        double2 temp[RY];
        T2 xl[RY][FDN / 2 + 1], xr[RY][FDN / 2 + 1];  // pairs at -2s and +2s of the row
        T2 ym[FDN + 1], yp[FDN + 1];
#pragma unroll
        for (int j = 0; j < RY; j++) {
          temp[j].x = (double)fut[j][0].x * c0;
          temp[j].y = (double)fut[j][0].y * c0;
          xl[j][0] = xr[j][0] = fut[j][0];
        }
#pragma unroll
        for (int k = 1; k <= FDN; k++) {
          ym[k] = *reinterpret_cast<const T2 *>(cp - k * P);
          yp[k] = *reinterpret_cast<const T2 *>(cp + (RY - 1 + k) * P);
          const T2 *rb = ring + (rz < k ? rz + RSLOT - k : rz - k) * RS;  // plane z - k
#pragma unroll
          for (int j = 0; j < RY; j++) {
            if (k & 1) {  // arms k and k + 1 of the pair reach the pairs at -(k + 1) and k + 1
              xl[j][(k + 1) / 2] = *reinterpret_cast<const T2 *>(cp + j * P - (k + 1));
              xr[j][(k + 1) / 2] = *reinterpret_cast<const T2 *>(cp + j * P + (k + 1));
            }
            // x - k, x + k of the pair's columns
            const T m0 = (k & 1) ? xl[j][(k + 1) / 2].y : xl[j][k / 2].x;
            const T p0 = (k & 1) ? xr[j][(k - 1) / 2].y : xr[j][k / 2].x;
            const T m1 = (k & 1) ? xl[j][(k - 1) / 2].x : xl[j][k / 2].y;
            const T p1 = (k & 1) ? xr[j][(k + 1) / 2].x : xr[j][k / 2].y;
            const T2 ylo = j >= k ? fut[j >= k ? j - k : 0][0] : ym[j >= k ? 1 : k - j];
            const T2 yhi = j + k < RY ? fut[j + k < RY ? j + k : 0][0] : yp[j + k < RY ? 1 : j + k - RY + 1];
            const T2 zm = rb[j * NT];
            const T s0 = m0 + p0 + ylo.x + yhi.x + zm.x + fut[j][k].x;
            const T s1 = m1 + p1 + ylo.y + yhi.y + zm.y + fut[j][k].y;
            temp[j].x += (double)s0 * a.coeff_lap[k];
            temp[j].y += (double)s1 * a.coeff_lap[k];
          }
        }
#pragma unroll
        for (int j = 0; j < RY; j++) {
          const int X = X0 + z * EP + j * a.ex;
          double2 vnl = make_double2(0.0, 0.0);
#pragma unroll
          for (int k = 0; k < KL; k++) {
            const unsigned i0 = lay_of(idc[j][0], k), i1 = lay_of(idc[j][1], k);
#pragma unroll
            for (int q = 0; q < PM; q++) {
              double2 ch;
              if constexpr (CHR) ch = chc[j][k];
              else ch = ok[j] ? chi_ld(j, k * PM + q, k, X) : make_double2(0.0, 0.0);
              vnl.x += pcur[SQB_IDX(i0 + q, a.n_gproj + PM, st)] * ch.x;
              vnl.y += pcur[SQB_IDX(i1 + q, a.n_gproj + PM, st)] * ch.y;
            }
          }
          v[j].x = (double)fut[j][0].x;
          v[j].y = (double)fut[j][0].y;
          hv[j].x = -0.5 * temp[j].x + ve[j].x * v[j].x + vnl.x;
          hv[j].y = -0.5 * temp[j].y + ve[j].y * v[j].y + vnl.y;
        }
      }
#pragma unroll
      for (int j = 0; j < RY; j++) {
        if (!ok[j]) continue;
        const int g = SQB_IDX(g0 + z * VP + j * NP, NW - 1, st);
        double2 o;
        if constexpr (SK == SK_ONES) {
          const unsigned par = par0 + j + z;
          o = make_double2(cv0 ? start_val(io.chk, par) : 0.0, cv1 ? start_val(io.chk, par + 1u) : 0.0);
        } else {
          T2 ot;
          if constexpr (SK == SK_LZF) {
            ot.x = cv0 ? (T)hv[j].x : T(0);
            ot.y = cv1 ? (T)hv[j].y : T(0);
            acc0 += v[j].x * v[j].x;
            acc0 += v[j].y * v[j].y;
            acc1 += v[j].x * hv[j].x;  // (v is zero in the pad column)
            acc1 += v[j].y * hv[j].y;
          } else {
            // sq.cpp:588, 615 divide by zee; the sweep multiplies by 1/zee
            // (one rounding apart, no FP64 division per point)
            double2 od;
            od.x = (hv[j].x - io.ca * v[j].x) * rcb - (double)q1[j].x;
            od.y = (hv[j].y - io.ca * v[j].y) * rcb - (double)q1[j].y;
            ot.x = cv0 ? (T)od.x : T(0);
            ot.y = cv1 ? (T)od.y : T(0);
          }
          __stcg(reinterpret_cast<T2 *>(io.out + g), ot);
          o.x = (double)ot.x;
          o.y = (double)ot.y;
          if constexpr (CHEB) {
            if (io.dbl) {
              acc0 += o.x * o.x;
              acc0 += o.y * o.y;
              acc1 += o.x * v[j].x;
              acc1 += o.y * v[j].y;
            }
            if constexpr (SK == SK_FD) {  // forces.cpp:414-456 (Ci / h^3 formed once per sweep)
              double2 dn;
              if (io.first) dq[j] = make_double2(v[j].x * ceh, v[j].y * ceh);  // (the input is e_c)
              dn.x = dq[j].x + o.x * cdh;
              dn.y = dq[j].y + o.y * cdh;
              __stcg(reinterpret_cast<double2 *>(io.dacc + g), dn);
            }
          }
          if (z == nl && ctr && j == cj) S.center_val = cc ? o.y : o.x;
          big = max(big, max((unsigned)__double2hiint(o.x) & 0x7fffffffu, (unsigned)__double2hiint(o.y) & 0x7fffffffu));
        }
        const int X = X0 + z * EP + j * a.ex;
        (void)X;
#pragma unroll
        for (int k = 0; k < KL; k++) {
#pragma unroll
          for (int q = 0; q < PM; q++) {
            double2 ch;
            if constexpr (CHR) ch = chc[j][k];
            else ch = chi_ld(j, k * PM + q, k, X);
            acd[j][k][q].x += ch.x * o.x;
            acd[j][k][q].y += ch.y * o.y;
            if constexpr (IND) {
              acw[j][k].x += ch.x * v[j].x;
              acw[j][k].y += ch.y * v[j].y;
            }
          }
        }
      }
      // a column that leaves a layer's ball after plane z flushes its partial
      // to the slot of (layer, z, column) and takes the next ball's coefficient
      unsigned long long chg = 0ull;
#pragma unroll
      for (int j = 0; j < RY; j++) chg |= (idc[j][0] ^ idn[j][0]) | (idc[j][1] ^ idn[j][1]);
      if (z + 1 < n && chg != 0ull) {
#pragma unroll
        for (int k = 0; k < KL; k++) {
          if (lay_of(chg, k) == 0u) continue;
#pragma unroll
          for (int j = 0; j < RY; j++) {
#pragma unroll
            for (int i = 0; i < 2; i++) {
              const unsigned was = lay_of(idc[j][i], k), now = lay_of(idn[j][i], k);
              if (was != now) {
                if (was != dummy) {
                  const int f = SQB_IDX((k * PM * n + z) * VP + g0 + j * NP + i, fset - (PM - 1) * NW, st);
#pragma unroll
                  for (int q = 0; q < PM; q++) fb[f + q * NW] = i ? acd[j][k][q].y : acd[j][k][q].x;
                  if constexpr (IND) fb[f + fset] = i ? acw[j][k].y : acw[j][k].x;
                }
#pragma unroll
                for (int q = 0; q < PM; q++) (i ? acd[j][k][q].y : acd[j][k][q].x) = 0.0;
                if constexpr (IND) (i ? acw[j][k].y : acw[j][k].x) = 0.0;
              }
            }
          }
        }
      }
    }
    // advance: ids, point data and the stencil input
#pragma unroll
    for (int j = 0; j < RY; j++) {
      if (z + 1 < n) {
        idc[j][0] = idn[j][0];
        idc[j][1] = idn[j][1];
      }
      load_ids(j, z + 2);
      load_point(j, z + 1);
      if constexpr (STENCIL) {
        ring[rz * RS + j * NT] = fut[j][0];  // plane z moves behind
#pragma unroll
        for (int s = 0; s < F - 1; s++) fut[j][s] = fut[j][s + 1];
        fut[j][F - 1] = next_in(j, z + FDN + 1);
        load_ops(j, z + FDN + 2);
      }
    }
    if constexpr (STENCIL) {
      if (z + 1 < n) pbar_wait(S, a.status, ph0 + (unsigned)z);
    }
    bz = bn;
    rz = rz == RSLOT - 1 ? 0 : rz + 1;
  }
  if (big >= 0x7ff00000u) atomicOr(a.status, ST_NONFINITE);
  if constexpr (STENCIL) {
    // every thread read ph0 before its first arrival, and thread 0 passed
    // every wait of this sweep
    if (tid == 0) S.pbar_phase = ph0 + (unsigned)(n - 1);
  }
  // balls that end at the window's last plane: the open partials; then every
  // ball's columns are summed
#pragma unroll
  for (int j = 0; j < RY; j++) {
    if (!ok[j]) continue;
#pragma unroll
    for (int k = 0; k < KL; k++) {
#pragma unroll
      for (int i = 0; i < 2; i++) {
        if (lay_of(idc[j][i], k) == dummy) continue;
        const int f = (k * PM * n + n - 1) * VP + g0 + j * NP + i;
#pragma unroll
        for (int q = 0; q < PM; q++) fb[f + q * NW] = i ? acd[j][k][q].y : acd[j][k][q].x;
        if constexpr (IND) fb[f + fset] = i ? acw[j][k].y : acw[j][k].x;
      }
    }
  }
  bar_sweep(NS);
  reduce_instances<PM, IND>(a, S, fb, warp, nwarp, lane);
  bar_sweep(NS);
}

// Sum of two values over the block into S.scal (deterministic).
static __device__ void sweep_sum2(Shared &S, double v0, double v1, int NS) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = NS >> 5;
  v0 = warp_sum(v0);
  v1 = warp_sum(v1);
  if (lane == 0) {
    S.red[warp][0] = v0;
    S.red[warp][1] = v1;
  }
  bar_sweep(NS);
  if (warp == 0) {
    double r0 = lane < nw ? S.red[lane][0] : 0.0;
    double r1 = lane < nw ? S.red[lane][1] : 0.0;
    r0 = warp_sum(r0);
    r1 = warp_sum(r1);
    if (lane == 0) {
      S.scal[0] = r0;
      S.scal[1] = r1;
    }
  }
  bar_sweep(NS);
}

// Sturm count: eigenvalues of the leading m x m tridiagonal (d, e) below x,
// from the sign changes of the characteristic-polynomial sequence
// p_i = (d_i - x) p_i-1 - e_i-1^2 p_i-2, rescaled by exact powers of two every
// eight rows (a row grows |p| by less than 2^64 here, far inside the range),
// which leaves every sign and rounding unchanged.  An exact zero counts as
// positive (a test point on an eigenvalue of a leading submatrix; the
// multisection's brackets tolerate the one-off count there).
static __device__ int sturm_count(const double *d, const double *e2, int m, double x) {
  double p0 = 1.0, p1 = d[0] - x;
  int cnt = p1 < 0.0;
  int i = 1;
  auto row = [&](int r) {
    const double p2 = (d[r] - x) * p1 - e2[r - 1] * p0;
    cnt += (p2 < 0.0) != (p1 < 0.0);
    p0 = p1;
    p1 = p2;
  };
  for (; i + 8 <= m; i += 8) {
#pragma unroll
    for (int r = 0; r < 8; r++) row(i + r);
    const double mx = fmax(fabs(p0), fabs(p1));
    if (mx > 0x1p+600) {
      p0 *= 0x1p-600;
      p1 *= 0x1p-600;
    } else if (mx < 0x1p-600 && mx > 0.0) {
      p0 *= 0x1p+600;
      p1 *= 0x1p+600;
    }
  }
  for (; i < m; i++) row(i);
  return cnt;
}

// Extreme eigenvalues of the m x m Lanczos tridiagonal (the quantities
// TridiagEigenSolve, sq.cpp:1094-1180, returns) into S.eig: the block's warps
// split into two groups, one per extreme, and each round every lane of a group
// evaluates a Sturm count at one of its 32 G points (G warps per group), so the
// bracket shrinks (32 G + 1)-fold per round, from the Gershgorin interval to
// four units in the last place.  All threads call it.
static __device__ void tridiag_extremes(Shared &S, int m) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
  const int G = nw / 2, N = 32 * G;
  const int g = warp < G ? 0 : (warp < 2 * G ? 1 : 2);
  const int gi = warp - g * G;
  // Gershgorin interval: the complete rows' part is kept by lanczos, the last
  // row has one neighbour.  Warm start from the previous (one row smaller)
  // tridiagonal's extremes: by interlacing the new smallest lies at or below
  // the old one and the new largest at or above it; the other end of each
  // bracket is the old extreme moved by four times its last change, which the
  // first round tests beside its inner points.
  const double rl = m > 1 ? fabs(S.bb[m - 2]) : 0.0;
  double glo = fmin(S.ger[0], S.aa[m - 1] - rl), ghi = fmax(S.ger[1], S.aa[m - 1] + rl);
  const double span = fmax(fabs(glo), fabs(ghi));
  glo -= 1e-14 * span + 1e-300;
  ghi += 1e-14 * span + 1e-300;
  bool first = S.warm != 0;
  if (tid == 0) {
    S.br[0][0] = S.br[1][0] = glo;
    S.br[0][1] = S.br[1][1] = ghi;
    if (first) {
      const double pad = 16.0 * 2.220446049250313e-16 * span;
      const double x0 = S.eig[0] - fmax(4.0 * S.wdel[0], 1e-9 * span), x1 = S.eig[1] + fmax(4.0 * S.wdel[1], 1e-9 * span);
      if (S.eig[0] + pad < ghi) S.br[0][1] = S.eig[0] + pad;
      if (S.eig[1] - pad > glo) S.br[1][0] = S.eig[1] - pad;
      S.br[0][0] = fmax(x0, glo);
      S.br[1][1] = fmin(x1, ghi);
    }
  }
  __syncthreads();
  auto active = [&](int k) {
    const double lo = S.br[k][0], hi = S.br[k][1];
    return hi - lo > 4.0 * 2.220446049250313e-16 * fmax(fabs(lo), fabs(hi)) + 1e-300;
  };
  for (int it = 0; it < 80; it++) {
    const bool a0 = first || active(0), a1 = first || active(1);
    if (!a0 && !a1) break;
    // points of a round: lo + w i / (N + 1), i = 1 .. N; in a warm first round
    // the guessed end is a point too: i = 0 .. N - 1 for the smallest (lo
    // guessed), i = 2 .. N + 1 for the largest (hi guessed)
    const int sh = first ? (g == 0 ? -1 : 1) : 0;
    const double inv = 1.0 / (double)(N + 1);
    if (g < 2 && (g == 0 ? a0 : a1)) {
      const double lo = S.br[g][0], w = S.br[g][1] - lo;
      const int i = gi * 32 + lane, j = i + 1 + sh;
      const int c = sturm_count(S.aa, S.b2, m, j == N + 1 ? S.br[g][1] : lo + w * ((double)j * inv));
      if (g == 0) {
        const unsigned below = __ballot_sync(0xffffffffu, c >= 1);
        if (lane == 0) S.wres[warp] = below ? gi * 32 + __ffs(below) - 1 : N;
      } else {
        const unsigned above = __ballot_sync(0xffffffffu, c < m);
        if (lane == 0) S.wres[warp] = above ? gi * 32 + 31 - __clz(above) : -1;
      }
    }
    __syncthreads();
    if (tid < 2 && (tid == 0 ? a0 : a1)) {
      const double lo = S.br[tid][0], hi = S.br[tid][1], w = hi - lo;
      if (tid == 0) {  // smallest: the first point with an eigenvalue below it
        const int s0 = first ? -1 : 0;
        int f = N;
        for (int v = 0; v < G; v++) f = min(f, S.wres[v]);
        if (f < N) S.br[0][1] = f + 1 + s0 == 0 ? lo : lo + w * ((double)(f + 1 + s0) * inv);
        if (f > 0) S.br[0][0] = f + s0 == 0 ? lo : lo + w * ((double)(f + s0) * inv);
        else if (first) S.br[0][0] = glo;  // an eigenvalue lies below the guess
      } else {  // largest: the last point with an eigenvalue above it
        const int s1 = first ? 1 : 0;
        int l = -1;
        for (int v = 0; v < G; v++) l = max(l, S.wres[G + v]);
        if (l >= 0) S.br[1][0] = l + 1 + s1 == N + 1 ? hi : lo + w * ((double)(l + 1 + s1) * inv);
        if (l < N - 1) S.br[1][1] = l + 2 + s1 == N + 1 ? hi : lo + w * ((double)(l + 2 + s1) * inv);
        else if (first) S.br[1][1] = ghi;  // an eigenvalue lies above the guess
      }
    }
    first = false;
    __syncthreads();
  }
  if (tid == 0) {
    S.eig[0] = 0.5 * (S.br[0][0] + S.br[0][1]);
    S.eig[1] = 0.5 * (S.br[1][0] + S.br[1][1]);
  }
  __syncthreads();
}

// The boxes of the replica balls meeting this node's window (the
// intersection test of nonlocal.cpp:66-108), their projector instances and
// the denominators.
static __device__ void setup_node(const SweepArgs &a, Shared &S) {
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
  const int n = a.n;
  if (tid == 0) S.n_ent = 0;
  __syncthreads();
  for (int base = 0; base < a.n_rep; base += nt) {
    const int r = base + tid;
    bool hit = false;
    int4 b = make_int4(0, 0, 0, 0);
    int x0 = 0, x1 = 0, y0 = 0, y1 = 0, z0 = 0, z1 = 0;
    if (r < a.n_rep) {
      b = a.rep_box[r];
      x0 = max((int)(short)(b.x & 0xffff), S.gi) - S.gi;
      x1 = min(b.x >> 16, S.gi + n - 1) - S.gi;
      y0 = max((int)(short)(b.y & 0xffff), S.gj) - S.gj;
      y1 = min(b.y >> 16, S.gj + n - 1) - S.gj;
      z0 = max((int)(short)(b.z & 0xffff), S.gk) - S.gk;
      z1 = min(b.z >> 16, S.gk + n - 1) - S.gk;
      hit = x0 <= x1 && y0 <= y1 && z0 <= z1;
    }
    const unsigned bal = __ballot_sync(0xffffffffu, hit);
    if (lane == 0) S.scan[warp] = __popc(bal);
    __syncthreads();
    if (tid == 0) {
      int s = 0;
      for (int w = 0; w < nw; w++) {
        const int v = S.scan[w];
        S.scan[w] = s;
        s += v;
      }
      S.scan[32] = s;
    }
    __syncthreads();
    if (hit) {
      const int pos = S.n_ent + S.scan[warp] + __popc(bal & ((1u << lane) - 1u));
      if (pos < MAXE) {
        S.e_x0[pos] = (short)x0;
        S.e_x1[pos] = (short)x1;
        S.e_y0[pos] = (short)y0;
        S.e_y1[pos] = (short)y1;
        S.e_z0[pos] = (short)z0;
        S.e_z1[pos] = (short)z1;
        S.e_k[pos] = (unsigned char)(b.w & 0xff);
        S.e_np[pos] = (unsigned char)((b.w >> 8) & 0xff);
        S.e_t[pos] = (unsigned char)((b.w >> 16) & 0xff);
        S.e_gpb[pos] = a.rep_gpb[r];
        S.e_r[pos] = r;
        S.e_atom[pos] = a.rep_atom ? a.rep_atom[r] : -1;
      } else {
        atomicOr(a.status, ST_CAPACITY);
      }
    }
    __syncthreads();
    if (tid == 0) S.n_ent = min(S.n_ent + S.scan[32], MAXE);
    __syncthreads();
  }
  if (tid == 0) {
    int pb = 0, ne = S.n_ent;
    for (int e = 0; e < ne; e++) {
      if (pb + S.e_np[e] > MAXP) {
        atomicOr(a.status, ST_CAPACITY);
        ne = e;
        break;
      }
      S.e_pb[e] = (short)pb;
      pb += S.e_np[e];
    }
    S.n_ent = ne;
    S.n_pi = pb;
  }
  __syncthreads();
  for (int e = 0; e < S.n_ent; e++)
    for (int q = tid; q < S.e_np[e]; q += nt) {
      const int p = S.e_pb[e] + q;
      S.pi_e[p] = (short)e;
      S.pi_g[p] = S.e_gpb[e] + q;
      S.p_den[p] = a.proj_denom[S.e_t[e] * MAXPROJ_TYPE + q];
      S.p_nxt[p] = 0.0;
    }
  __syncthreads();
}

// chi^T e_c of every instance (the projector values at the window centre;
// zero for balls that do not hold it) into pw_cur, and c = chi^T e_c / Denom
// into the gather array.
static __device__ void centre_projections(const SweepArgs &a, Shared &S, double *pcur) {
  const int nl = a.nloc;
  const int X = ((S.gk + nl) * a.ey + (S.gj + nl)) * a.ex + S.gi + nl;
  for (int p = threadIdx.x; p < S.n_pi; p += blockDim.x) {
    const int e = S.pi_e[p], q = p - S.e_pb[e], k = S.e_k[e];
    const bool in = S.e_x0[e] <= nl && nl <= S.e_x1[e] && S.e_y0[e] <= nl && nl <= S.e_y1[e] && S.e_z0[e] <= nl &&
                    nl <= S.e_z1[e];
    const double c = in ? a.lay_chi[(k * a.pmax + q) * (int)a.evol + X] : 0.0;
    S.pw_cur[p] = c;
    S.pw_prev[p] = 0.0;
    pcur[S.pi_g[p]] = c / S.p_den[p];
  }
  __syncthreads();
}

// c_J = chi_J^T w / Denom_J of the last sweep's output into the gather array.
static __device__ void rotate(Shared &S, double *pcur) {
  for (int p = threadIdx.x; p < S.n_pi; p += blockDim.x) pcur[S.pi_g[p]] = S.p_nxt[p] / S.p_den[p];
  __syncthreads();
}

static __device__ void count_proj_points(const SweepArgs &a, Shared &S, long long steps, int cheb) {
  if (threadIdx.x != 0 || a.proj_points == nullptr) return;
  unsigned long long full = 0, win = 0;
  for (int e = 0; e < S.n_ent; e++) {
    const unsigned long long Sd = 2ull * a.typ_nlocc[S.e_t[e]] + 1ull;
    full += (unsigned long long)S.e_np[e] * Sd * Sd * Sd;
    win += (unsigned long long)S.e_np[e] * (S.e_x1[e] - S.e_x0[e] + 1) * (S.e_y1[e] - S.e_y0[e] + 1) *
           (S.e_z1[e] - S.e_z0[e] + 1);
  }
  atomicAdd(a.proj_points, full * (unsigned long long)steps);
  if (cheb) atomicAdd(a.proj_points + 1, full * (unsigned long long)steps);
  atomicAdd(a.proj_points + 2, win * (unsigned long long)steps);
}

// What lanczos and moments need of a kernel's tile: its sweep and the layout of
// its window vectors (rows of `cols` values, window column x at x + shift).
template <int PM_, int RY, int NT>
struct PairTile {
  static constexpr int PM = PM_;
  static __device__ __forceinline__ int cols(int n) { return pair_cols(n); }
  static __device__ __forceinline__ int shift(const Shared &S) { return S.gi & 1; }
  template <typename T, int SK>
  static __device__ __forceinline__ void run(const SweepArgs &a, Shared &S, unsigned char *dyn, const IO<T> &io,
                                             double &acc0, double &acc1) {
    sweep<T, PM, SK, RY, NT>(a, S, dyn, io, acc0, acc1);
  }
};

// The node's unit vector e_c, and the scaled Lanczos start vector, into a
// window vector (pad columns zero).
template <class Tile, typename T>
static __device__ void unit_vector(const SweepArgs &a, Shared &S, T *v) {
  const int NP = Tile::cols(a.n), nw = a.n * a.n * NP, nl = a.nloc;
  const int c = (nl * a.n + nl) * NP + nl + Tile::shift(S);
  __syncthreads();
  for (int i = threadIdx.x; i < nw; i += blockDim.x) v[i] = (T)(i == c ? 1.0 : 0.0);
  __syncthreads();
}
template <class Tile, typename T>
static __device__ void start_vector(const SweepArgs &a, Shared &S, T *v, double scale) {
  const int n = a.n, NP = Tile::cols(n), nw = n * n * NP, sh = Tile::shift(S);
  __syncthreads();
  for (int i = threadIdx.x; i < nw; i += blockDim.x) {
    const int row = i / NP, x = i - row * NP - sh;  // row = z n + y, of the parity of z + y
    v[i] = (T)(x >= 0 && x < n ? scale * start_val(a.lz_chk, row + x) : 0.0);
  }
  __syncthreads();
}

constexpr int LANCZOS_LEFT = 2;  // S.stop of a run left to another kernel (redo_at)

// Lanczos bounds (sq.cpp:965-1092) in storage precision T, or (LQ) bounds and
// moments from one FP64 Lanczos run started at e_c.  Sweep m applies H to the
// unnormalised W_m = w_m-1 (v_m = s_m W_m), formed while it is loaded from the
// previous sweep's output Y_m-1 = H W_m-1 and the two previous W; it yields
// <W_m, W_m> = b_m-1^2 and <W_m, H W_m> = a_m b_m-1^2, so after sweep m the
// tridiagonal T_m+1 is complete and the reference's convergence test (both
// extremes moved by no more than the tolerance, at most 500 steps) applies.
// The projections chi^T W_m+1 the next gather needs follow from the recurrence
// on the dot products of the sweep's output.
template <class Tile, typename T, bool LQ>
__device__ void lanczos(const SweepArgs &a, Shared &S, unsigned char *dyn, double *pcur, double &lmin_out,
                        double &lmax_out, int &rows_out) {
  constexpr int PM = Tile::PM;
  const int tid = threadIdx.x;
  const double nw = (double)a.n * a.n * a.n;
  T *Y = slot<T>(a, 0);
  T *Wv[2] = {slot<T>(a, 1), slot<T>(a, 2)};
  const double chk = a.lz_chk;
  const double s0 = LQ ? 1.0 : 1.0 / sqrt(nw * (1.0 + chk * chk) + 2.0 * chk);
  const int kmin = a.npl / 2 + 1;
  double d0 = 0.0, d1 = 0.0;
  if constexpr (LQ) {
    unit_vector<Tile>(a, S, Y);
    centre_projections(a, S, pcur);  // W_0 = e_c
  } else {
    start_vector<Tile>(a, S, Y, s0);
    // chi^T W_0 for W_0 = (1 + chk (-1)^(x+y+z)) / norm (sq.cpp:538-546, 993-1004
    // with chk = 0)
    IO<T> io;
    io.chk = chk;
    Tile::template run<T, SK_ONES>(a, S, dyn, io, d0, d1);
    __syncthreads();
    for (int p = tid; p < S.n_pi; p += blockDim.x) {
      S.pw_cur[p] = s0 * S.p_nxt[p];
      S.pw_prev[p] = 0.0;
      pcur[S.pi_g[p]] = S.pw_cur[p] / S.p_den[p];
    }
  }
  if (tid == 0) {
    S.stop = 0;
    S.count = 0;
    S.eprev[0] = S.eprev[1] = 0.0;
    S.warm = 0;
    S.ger[0] = 1e300;
    S.ger[1] = -1e300;
  }
  __syncthreads();
  double a_prev = 0.0, s_prev = 1.0, bs_prev = 0.0;
  for (int m = 0;; m++) {
    IO<T> io;
    io.out = Y;
    io.wout = Wv[m & 1];
    if (m == 0) {  // W_0 = 1 (Y - 0 W1) - 0 W2 from the start vector in Y
      io.vin = io.p1 = io.p2 = Y;
    } else {
      io.vin = Y;
      io.p1 = Wv[(m - 1) & 1];
      io.p2 = m >= 2 ? Wv[m & 1] : Wv[(m - 1) & 1];  // no third term in the first step (sq.cpp:1006-1014)
      io.s1 = s_prev;
      io.ca = a_prev;
      io.cb = bs_prev;
    }
    d0 = 0.0;
    d1 = 0.0;
    Tile::template run<T, SK_LZF>(a, S, dyn, io, d0, d1);
    sweep_sum2(S, d0, d1, a.nsweep);
    // b_m-1 = |W_m| and a_m = <W_m, H W_m> / b_m-1^2 (W_0 is normalised)
    const double bm = m == 0 ? 1.0 : sqrt(S.scal[0]);
    const double am = S.scal[1] / (bm * bm);
    const double sm = 1.0 / bm;
    if (tid == 0) {
      S.aa[m] = am;
      if (m > 0) {
        S.bb[m - 1] = bm;
        S.b2[m - 1] = bm * bm;
        const double r = bm + (m > 1 ? S.bb[m - 2] : 0.0);  // row m - 1 is complete
        S.ger[0] = fmin(S.ger[0], S.aa[m - 1] - r);
        S.ger[1] = fmax(S.ger[1], S.aa[m - 1] + r);
      }
    }
    __syncthreads();
    // after sweep m the tridiagonal has m + 1 rows (complete from m = 1; the
    // quadrature form follows its extremes from npl/2 rows on, so that the run
    // can stop at the npl/2 + 1 rows its moments need)
    const bool solve = LQ ? (m + 2 >= kmin) : (m >= 1);
    if (solve) {
      tridiag_extremes(S, m + 1);
      if (tid == 0) {
        const double dl = fabs(S.eig[0] - S.eprev[0]), dm = fabs(S.eig[1] - S.eprev[1]);
        S.eprev[0] = S.eig[0];
        S.eprev[1] = S.eig[1];
        S.wdel[0] = S.warm ? dl : 0.0;  // (the first solve's change is against zero)
        S.wdel[1] = S.warm ? dm : 0.0;
        S.warm = 1;
        const bool conv = !(dl > a.lanczos_tol || dm > a.lanczos_tol);
        if constexpr (LQ) {
          S.count = m + 1;  // rows of T; the first solve only sets the previous extremes
          S.stop = (m + 2 > kmin && conv) || S.count >= LANCZOS_MAX_ITER;
        } else {
          S.count = m;  // the reference's count after this step
          S.stop = conv || S.count >= LANCZOS_MAX_ITER;
          if constexpr (Tile::PM > 1 && std::is_same<T, double>::value) {
            if (!S.stop && a.redo_count && m >= a.redo_at) S.stop = LANCZOS_LEFT;
          }
        }
        if (S.count >= LANCZOS_MAX_ITER) atomicOr(a.status, ST_LANCZOS_MAXITER);
      }
      __syncthreads();
      if (S.stop) break;
    }
    // chi^T W_m+1 = s_m (chi^T Y_m - a_m chi^T W_m) - b_m-1 s_m-1 chi^T W_m-1.
    // With input dots the two older terms are the exact dot products of the
    // stored W_m and W_m-1, so only this step's rounding enters the gather of
    // the next sweep.  Without them (several projectors per layer slot) they
    // are the recurrence's own earlier values, whose rounding the three-term
    // recurrence amplifies like the Lanczos polynomials at 0: harmless for the
    // usual step counts when 0 lies inside the window's spectrum, growing
    // exponentially in the step count when it does not.
    const double bs_cur = m == 0 ? 0.0 : bm * s_prev;
    for (int p = tid; p < S.n_pi; p += blockDim.x) {
      const double wm = input_dots(PM) ? S.p_in[p] : S.pw_cur[p];
      const double nx = sm * (S.p_nxt[p] - am * wm) - bs_cur * S.pw_prev[p];
      S.pw_prev[p] = wm;
      S.pw_cur[p] = nx;
      pcur[S.pi_g[p]] = nx / S.p_den[p];
    }
    __syncthreads();
    a_prev = am;
    bs_prev = bs_cur;
    s_prev = sm;
  }
  lmin_out = S.eig[0] - a.lanczos_tol;
  lmax_out = S.eig[1] + a.lanczos_tol;
  rows_out = S.count;
}

// Chebyshev moments mu_j = e_c^T T_j((H - chi)/zee) e_c / h^3 (sq.cpp:564-655).
template <class Tile>
__device__ void moments(const SweepArgs &a, Shared &S, unsigned char *dyn, double *pcur, double chi, double zee,
                        double *mu) {
  double *B0 = slot<double>(a, 0), *B1 = slot<double>(a, 1);
  double d0 = 0.0, d1 = 0.0;
  centre_projections(a, S, pcur);
  unit_vector<Tile>(a, S, B0);
  {  // t_1 = (H e_c - chi e_c) / zee
    IO<double> io;
    io.vin = B0;
    io.first = 1;
    io.out = B1;
    io.ca = chi;
    io.cb = zee;
    Tile::template run<double, SK_CH>(a, S, dyn, io, d0, d1);
  }
  __syncthreads();
  rotate(S, pcur);
  const double htemp = S.center_val;
  if (threadIdx.x == 0) {
    mu[0] = (double)(1.0 / a.h3);
    mu[1] = (double)(htemp / a.h3);
  }
  double *t0 = B0, *t1 = B1;
  const int q1 = (int)rint(0.25 * a.npl), q2 = (int)rint(0.5 * a.npl);
  for (int nq = 2; nq <= q2; nq++) {
    {
      IO<double> io;
      io.vin = t1;
      io.p1 = t0;
      io.out = t0;
      io.ca = chi;
      io.cb = zee;
      io.dbl = nq > q1;
      d0 = 0.0;
      d1 = 0.0;
      Tile::template run<double, SK_CH>(a, S, dyn, io, d0, d1);
      if (nq > q1) sweep_sum2(S, d0, d1, a.nsweep);
    }
    __syncthreads();
    rotate(S, pcur);
    if (threadIdx.x == 0) {
      mu[nq] = (double)(S.center_val / a.h3);
      if (nq > q1) {
        mu[2 * nq] = (double)((2 * S.scal[0] - 1) / a.h3);
        mu[2 * nq - 1] = (double)((2 * S.scal[1] - htemp) / a.h3);
      }
    }
    double *tt = t0;
    t0 = t1;
    t1 = tt;
  }
}

// Sum of three values over the block into S.scal2 (deterministic).
static __device__ void sweep_sum3(Shared &S, double v0, double v1, double v2) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  v0 = warp_sum(v0);
  v1 = warp_sum(v1);
  v2 = warp_sum(v2);
  if (lane == 0) {
    S.red3[warp][0] = v0;
    S.red3[warp][1] = v1;
    S.red3[warp][2] = v2;
  }
  __syncthreads();
  if (warp == 0) {
    double r0 = lane < nw ? S.red3[lane][0] : 0.0;
    double r1 = lane < nw ? S.red3[lane][1] : 0.0;
    double r2 = lane < nw ? S.red3[lane][2] : 0.0;
    r0 = warp_sum(r0);
    r1 = warp_sum(r1);
    r2 = warp_sum(r2);
    if (lane == 0) {
      S.scal2[0] = r0;
      S.scal2[1] = r1;
      S.scal2[2] = r2;
    }
  }
  __syncthreads();
}

// ForcesNonLocal for one node (forces.cpp:318-578): the density-matrix column
// D = sum_k Ci_k T_k((H - chi)/zee) e_c / h^3 by the full npl-step Chebyshev
// recursion (vectors in storage precision T, D in FP64, slot 2 of the
// scratch), then, on each ball that holds the window centre, the FD gradient
// of D (zero outside the window) contracted with the replica's projectors:
// f = -4 h^3 sum_q (chi_q . grad D) chi_q(centre) / Denom_q, into the node's
// force slots (atom, fx, fy, fz).
template <typename T, int PM, int RY, int NT>
__device__ void node_forces(const SweepArgs &a, Shared &S, unsigned char *dyn, double *pcur, double chi,
                            double zee, const double *ci, double *fslot) {
  T *B0 = slot<T>(a, 0), *B1 = slot<T>(a, 1);
  double *D = slot<double>(a, 2);
  double d0 = 0.0, d1 = 0.0;
  unit_vector<PairTile<PM, RY, NT>>(a, S, B0);
  centre_projections(a, S, pcur);
  {  // t_1 = (H e_c - chi e_c) / zee; D = e_c Ci_0 / h^3 + t_1 Ci_1 / h^3
    IO<T> io;
    io.vin = B0;
    io.first = 1;
    io.out = B1;
    io.ca = chi;
    io.cb = zee;
    io.dacc = D;
    io.ce = ci[0];
    io.cd = ci[1];
    sweep<T, PM, SK_FD, RY, NT>(a, S, dyn, io, d0, d1);
  }
  __syncthreads();
  rotate(S, pcur);
  T *t0 = B0, *t1 = B1;
  for (int nq = 2; nq <= a.npl; nq++) {  // t_nq = 2 (H - chi)/zee t_nq-1 - t_nq-2; D += t_nq Ci_nq / h^3
    IO<T> io;
    io.vin = t1;
    io.p1 = t0;
    io.out = t0;
    io.ca = chi;
    io.cb = zee;
    io.dacc = D;
    io.cd = ci[nq];
    sweep<T, PM, SK_FD, RY, NT>(a, S, dyn, io, d0, d1);
    __syncthreads();
    rotate(S, pcur);
    T *tt = t0;
    t0 = t1;
    t1 = tt;
  }
  __threadfence_block();
  __syncthreads();
  const int n = a.n, nl = a.nloc, NP = pair_cols(n), VP = n * NP, sh = S.gi & 1, EV = (int)a.evol;
  int slotc = 0;
  for (int e = 0; e < S.n_ent; e++) {
    if (nl < S.e_x0[e] || nl > S.e_x1[e] || nl < S.e_y0[e] || nl > S.e_y1[e] || nl < S.e_z0[e] || nl > S.e_z1[e])
      continue;
    const int x0 = S.e_x0[e], y0 = S.e_y0[e], z0 = S.e_z0[e];
    const int bx = S.e_x1[e] - x0 + 1, by = S.e_y1[e] - y0 + 1, bz = S.e_z1[e] - z0 + 1, vol = bx * by * bz;
    const int k = S.e_k[e];
    double fx = 0.0, fy = 0.0, fz = 0.0;
    for (int q = 0; q < S.e_np[e]; q++) {
      const double *U = a.lay_chi + (size_t)(k * PM + q) * EV;
      double ax = 0.0, ay = 0.0, az = 0.0;
      for (int i = threadIdx.x; i < vol; i += blockDim.x) {
        const int x = x0 + i % bx, y = y0 + (i / bx) % by, z = z0 + i / (bx * by);
        const int w = SQB_IDX(z * VP + y * NP + x + sh, n * VP, a.status);
        double gx = 0.0, gy = 0.0, gz = 0.0;
        for (int kk = 1; kk <= FDN; kk++) {
          const double xm = x - kk >= 0 ? D[w - kk] : 0.0, xp = x + kk < n ? D[w + kk] : 0.0;
          const double ym = y - kk >= 0 ? D[w - kk * NP] : 0.0, yp = y + kk < n ? D[w + kk * NP] : 0.0;
          const double zm = z - kk >= 0 ? D[w - kk * VP] : 0.0, zp = z + kk < n ? D[w + kk * VP] : 0.0;
          gx += (-xm + xp) * a.coeff_grad[kk];
          gy += (-ym + yp) * a.coeff_grad[kk];
          gz += (-zm + zp) * a.coeff_grad[kk];
        }
        const double u = U[SQB_IDX(((S.gk + z) * a.ey + (S.gj + y)) * a.ex + S.gi + x, EV, a.status)];
        ax += u * gx;
        ay += u * gy;
        az += u * gz;
      }
      sweep_sum3(S, ax, ay, az);
      const double uc = U[((S.gk + nl) * a.ey + (S.gj + nl)) * a.ex + S.gi + nl];
      const double den = S.p_den[S.e_pb[e] + q];
      fx += S.scal2[0] / den * uc;
      fy += S.scal2[1] / den * uc;
      fz += S.scal2[2] / den * uc;
    }
    if (threadIdx.x == 0) {
      if (slotc < FSLOTS) {
        double *o = fslot + 4 * slotc;
        o[0] = (double)S.e_atom[e];
        o[1] = -4 * fx * a.h3;
        o[2] = -4 * fy * a.h3;
        o[3] = -4 * fz * a.h3;
      } else {
        atomicOr(a.status, ST_FSLOTS);
      }
    }
    slotc++;
    __syncthreads();
  }
  count_proj_points(a, S, a.npl, 1);
}

// The force pass over the listed nodes (bounds from chi, zee; Ci from ci).
template <int PM, typename T, int MAXT, int RY, int MINB>
__global__ void __launch_bounds__(MAXT, MINB) sweep_force_kernel(SweepArgs a) {
  extern __shared__ __align__(128) unsigned char smem[];
  Shared &S = *reinterpret_cast<Shared *>(smem);
  unsigned char *dyn = smem + shared_fixed();
  double *pcur = reinterpret_cast<double *>(dyn + planes_bytes(a.n, RY) + ring_bytes(MAXT, RY));
  for (int i = threadIdx.x; i < a.n_gproj + PM; i += blockDim.x) pcur[i] = 0.0;  // [n_gproj..]: the empty id
  pbar_setup(S);
  zero_planes(a, dyn, RY);
  for (;;) {
    if (threadIdx.x == 0) {
      const int q = atomicAdd(a.counter, 1);
      S.qidx = q;
      S.node = q < a.n_list ? a.node_list[q] : -1;
      if (S.node >= 0) {
        S.gi = S.node % a.np[0];
        S.gj = (S.node / a.np[0]) % a.np[1];
        S.gk = S.node / (a.np[0] * a.np[1]);
      }
    }
    __syncthreads();
    const int node = S.node;
    if (node < 0) break;
    double *fs = a.fslots + (size_t)S.qidx * FSLOTS * 4;
    for (int i = threadIdx.x; i < FSLOTS * 4; i += blockDim.x) fs[i] = (i % 4 == 0) ? -1.0 : 0.0;
    setup_node(a, S);
    node_forces<T, PM, RY, MAXT>(a, S, dyn, pcur, a.chi[node], a.zee[node], a.ci + (size_t)node * (a.npl + 1), fs);
    __syncthreads();
  }
}

// Moments of the quadrature form: mu_j = e_1^T T_j((T_k - chi)/zee) e_1 / h^3
// on the k-row tridiagonal (one warp, k-vectors in the free window slots).
static __device__ void quadrature_moments(const SweepArgs &a, Shared &S, int k, double chi, double zee, double *mu) {
  if (threadIdx.x >= 32) return;
  const int lane = threadIdx.x;
  double *v0 = slot<double>(a, 0), *v1 = slot<double>(a, 1), *v2 = slot<double>(a, 2);
  for (int i = lane; i < k; i += 32) {
    v0[i] = i == 0 ? 1.0 : 0.0;
    v1[i] = i == 0 ? (S.aa[0] - chi) / zee : (i == 1 ? S.bb[0] / zee : 0.0);
  }
  __syncwarp();
  if (lane == 0) {
    mu[0] = 1.0 / a.h3;
    mu[1] = v1[0] / a.h3;
  }
  for (int j = 1; j < a.npl; j++) {
    for (int i = lane; i < k; i += 32) {
      double t = (S.aa[i] - chi) / zee * v1[i];
      if (i > 0) t += S.bb[i - 1] / zee * v1[i - 1];
      if (i + 1 < k) t += S.bb[i] / zee * v1[i + 1];
      v2[i] = 2.0 * t - v0[i];
    }
    __syncwarp();
    if (lane == 0) mu[j + 1] = v2[0] / a.h3;
    double *tt = v0;
    v0 = v1;
    v1 = v2;
    v2 = tt;
    __syncwarp();
  }
}

// FORM: 0 FP64, 1 FP32-mixed, 2 Lanczos quadrature.  MAXT bounds the block,
// which sets the register budget per thread.
template <int PM, int FORM, int MAXT, int RY, int MINB>
__global__ void __launch_bounds__(MAXT, MINB) sweep_kernel(SweepArgs a) {
  using Tile = PairTile<PM, RY, MAXT>;
  extern __shared__ __align__(128) unsigned char smem[];
  Shared &S = *reinterpret_cast<Shared *>(smem);
  unsigned char *dyn = smem + shared_fixed();
  double *pcur = reinterpret_cast<double *>(dyn + planes_bytes(a.n, RY) + ring_bytes(MAXT, RY));
  for (int i = threadIdx.x; i < a.n_gproj + PM; i += blockDim.x) pcur[i] = 0.0;  // [n_gproj..]: the empty id
  pbar_setup(S);
  zero_planes(a, dyn, RY);
  for (;;) {
    if (threadIdx.x == 0) {
      const int q = atomicAdd(a.counter, 1);
      S.qidx = q;
      S.node = q < a.n_list ? a.node_list[q] : -1;
      if (S.node >= 0) {
        S.gi = S.node % a.np[0];
        S.gj = (S.node / a.np[0]) % a.np[1];
        S.gk = S.node / (a.np[0] * a.np[1]);
      }
    }
    __syncthreads();
    const int node = S.node;
    if (node < 0) break;
    setup_node(a, S);
    double lmin = 0.0, lmax = 0.0;
    int rows = 0;
    double *mu = a.rho_pj + (size_t)node * (a.npl + 1);
    if constexpr (FORM == 2) {
      lanczos<Tile, double, true>(a, S, dyn, pcur, lmin, lmax, rows);
      const double chi = 0.5 * (lmax + lmin), zee = 0.5 * (lmax - lmin);
      if ((long long)rows <= (long long)a.n * a.n * a.n) quadrature_moments(a, S, rows, chi, zee, mu);
      else if (threadIdx.x == 0) atomicOr(a.status, ST_CAPACITY);
      count_proj_points(a, S, rows, 0);
      rows -= 1;  // reported as Lanczos iterations: matvecs = iterations + 1
    } else {
      using TL = typename std::conditional<FORM == 1, float, double>::type;
      if (FORM == 1) zero_planes(a, dyn, RY);  // FP32 values next
      lanczos<Tile, TL, false>(a, S, dyn, pcur, lmin, lmax, rows);
      if constexpr (FORM == 0 && PM > 1) {
        if (S.stop == LANCZOS_LEFT) {
          if (threadIdx.x == 0) a.redo_list[atomicAdd(a.redo_count, 1)] = node;
          __syncthreads();
          continue;
        }
      }
      const double chi = (lmax + lmin) / 2, zee = (lmax - lmin) / 2;  // sq.cpp:564-565
      count_proj_points(a, S, rows + 1, 0);
      // moments stay FP64 in both forms: FP32 storage of the Chebyshev vectors
      // grows a rounding error injected at step i like (k - i) by step k
      if (FORM == 1) zero_planes(a, dyn, RY);  // FP64 values next
      moments<Tile>(a, S, dyn, pcur, chi, zee, mu);
      count_proj_points(a, S, a.npl / 2, 1);
    }
    if (threadIdx.x == 0) {
      a.chi[node] = (lmax + lmin) / 2;
      a.zee[node] = (lmax - lmin) / 2;
      if (a.lmin) a.lmin[node] = lmin;
      if (a.lmax) a.lmax[node] = lmax;
      if (a.lanczos_iters) a.lanczos_iters[node] = rows;
    }
    __syncthreads();
  }
}

// Tiles: a pair of columns and one row per thread, and a launch bound, which
// sets the registers per thread.  More rows share their y-arm loads and issue
// 20% fewer instructions per point, but leave fewer warps to hide latency.  Two
// rows, 8 warps of 255 registers against 16 of 128 (B200, 288 nodes of 31^3
// windows, FP64): 25.4 against 20.8 ms; 27^3: 23.4 against 16.6 ms.  Three rows
// (448 nodes, npl 64, FP64 step of Al): 7.5 against 1.6 ms at 9^3, 32 against 12
// at 21^3, 76 against 31 at 31^3, 94 against 55 at 33^3, and 1.4 to 10 times
// longer in the other forms, the forces, the adjoint and LiH.  The bounds follow
// the registers a warp count leaves (39^3: 124.7 ms at a bound of 896 and 72
// registers, 144.5 at 1024 and 64).  Shared memory holds three CTAs on an SM at
// 9^3, two from 11^3 to 19^3 (17^3: 82 KB each); fewer registers for the same two
// cost time (17^3, 1000 nodes: 13.3 ms at 112, 9.6 at 168).  From 23^3 on one CTA
// keeps 168 registers: 14.6, 17.6 and 20.0 ms at 23^3, 25^3 and 27^3 (448 nodes
// as above), against 24.4, 30.5 and 38.6 for two CTAs of 80.  The forces and the
// adjoint take the same tiles.
constexpr int TILE_RY = 1;
constexpr int TILE_N_MAX = 43;  // widest window
// Launch bound of the tile (and the ring's stride).
inline int tile_bound(int n) {
  const int t = sweep_threads_of(n, TILE_RY);
  return t <= 64 ? 64 : t <= 192 ? 192 : t <= 384 ? 384 : t <= 512 ? 512 : t <= 640 ? 640 : t <= 768 ? 768 : t <= 896 ? 896 : 1024;
}
template <class K>
const void *pick_tile(int n) {
  if (n > TILE_N_MAX) return nullptr;
  const int m = tile_bound(n);
  return m == 64    ? K::template get<64, 3>()
         : m == 192 ? K::template get<192, 2>()
         : m == 384 ? K::template get<384, 1>()
         : m == 512 ? K::template get<512, 1>()
         : m == 640 ? K::template get<640, 1>()
         : m == 768 ? K::template get<768, 1>()
         : m == 896 ? K::template get<896, 1>()
                    : K::template get<1024, 1>();
}
// Shared-memory limit of a kernel for a launch and, on request, its resident
// CTAs per SM; tile_setup: of a default-tile kernel for the launch `a`.
cudaError_t kernel_setup(const void *kernel, int threads, size_t smem, int *per_sm);
cudaError_t tile_setup(const void *kernel, const SweepArgs &a, int *per_sm);

}  // namespace sweep
}  // namespace sqb

// Sweep kernel with one window column per thread: the nodes of systems with up
// to three projectors per ball whose FP64 Lanczos runs are long.
//
// A run past about 6.5 window edges has lost the orthogonality of its vectors
// (LiH at h = 0.386, 33^3 windows: 80 to 321 steps, one node in twelve past 198).
// Where it stops on a plateau of the smallest eigenvalue, the accepted bound
// then depends on the rounding of every sum before it: relative noise of 1e-16
// on the vectors of a plain FP64 run with exact projections moves it by up to
// 1e-6 Ha, the stop itself, and the moments of the block by 2e-7.  No order of
// the sums is better than another there, but a caller's results should not
// change with the tile that is fastest.  So the column-pair kernel
// (sqb_sweep.cuh) leaves such nodes to a second launch, whose sums keep the
// order these bounds have always come from: of this kernel where first-fit
// layers cover the system, of the plane-streaming kernel where they do not.
// Measured on the B200, FP64 step of 64-atom LiH, 400 nodes of 33^3 windows:
// 400 to 808 ms all on the plane-streaming kernel, 180 (no long run) to 586 with
// the long runs there, 145 to 240 on column pairs alone.
//
// The plane loop is that of sqb_sweep.cuh without the pairs: window vectors of
// n^3 values, a thread per column and RY adjacent rows, the stencil's planes
// ahead in registers and behind in the thread's slots of a shared ring, three
// plane buffers under the split barrier.  The projector values of a point (up
// to twelve) are loaded where they are used: kept in registers they would
// spill.
#include "sqb_sweep.cuh"

namespace sqb {

namespace {

using namespace sweep;

constexpr int CPM = 3;    // projectors per layer slot
constexpr int CRSLOT = 8; // ring slots (a power of two above FDN)

__host__ __device__ constexpr int col_pitch(int n) { return n + 2 * FDN; }
// NPLANE halo'd planes, plus ry - 1 rows of slack: the shared y-arm loads of
// a row group whose last rows lie beyond the window read up to ry - 1 rows
// past the plane (into values that are not used).
__host__ __device__ inline size_t col_planes_bytes(int n, int ry) {
  const int P = col_pitch(n);
  return ((size_t)(NPLANE * P * P + (ry - 1) * P + 8) * sizeof(double) + 127) & ~size_t(127);
}
__host__ __device__ inline size_t col_ring_bytes(int nsweep, int ry) {
  return ((size_t)CRSLOT * ry * nsweep * sizeof(double) + 127) & ~size_t(127);
}
// Windows up to 32 wide give each row group a warp of its own (lane = column),
// so its shared-plane loads are one contiguous run; wider windows pack the
// columns densely.
__host__ __device__ inline int col_threads(int n, int ry) {
  const int groups = (n + ry - 1) / ry;
  const int t = n <= 32 ? 32 * groups : ((n * groups + 31) / 32) * 32;
  return t < 64 ? 64 : t;  // two warps at least: the multisection's two extremes
}

// Sum of one projector instance's flushed column partials over its box's
// columns, at the slots of its ball's last window plane (one warp, fixed
// order), into p_nxt.
__device__ __forceinline__ void col_reduce(const SweepArgs &a, Shared &S, const double *fb, int p, int lane) {
  const int e = S.pi_e[p], q = p - S.e_pb[e], k = S.e_k[e];
  const int n = a.n, n2 = n * n;
  const int x0 = S.e_x0[e], y0 = S.e_y0[e];
  const int bx = S.e_x1[e] - x0 + 1, by = S.e_y1[e] - y0 + 1, cnt = bx * by;
  const int base = ((k * CPM + q) * n + S.e_z1[e]) * n2 + y0 * n + x0, set = KL * CPM * n * n2;
  const double *f = fb + base;
  (void)set;
  double s = 0.0;
#pragma unroll 4
  for (int i = lane; i < cnt; i += 32) {
    const int yy = i / bx, xx = i - yy * bx;
    const int o = SQB_IDX(base + yy * n + xx, set, a.status) - base;
    s += f[o];
  }
  s = warp_sum(s);
  if (lane == 0) S.p_nxt[p] = s;
}

// One sweep over the window's z-planes (all threads of the block).
template <int SK, int RY>
__device__ __forceinline__ void col_sweep(const SweepArgs &a, Shared &S, unsigned char *dyn, const IO<double> &io,
                                          double &acc0, double &acc1) {
  constexpr bool STENCIL = SK != SK_ONES;
  constexpr int F = FDN + 1;  // planes held in registers: the centre and the FDN ahead
  const int n = a.n, n2 = n * n, P = col_pitch(n), P2 = P * P;
  const int tid = threadIdx.x, NS = a.nsweep, lane = tid & 31, warp = tid >> 5, nwarp = NS >> 5;
  const int nrow = (n + RY - 1) / RY;
  const bool lanes = n <= 32;
  const int tx = lanes ? (tid & 31) : tid % n, tg = lanes ? (tid >> 5) : tid / n;
  const bool tv = tx < n && tg < nrow;
  const int x = tv ? tx : 0, yb = tv ? tg * RY : 0;
  const int nl = a.nloc, gc = (nl * n + nl) * n + nl;  // window index of the centre
  const int EP = a.ex * a.ey, EV = (int)a.evol;        // the extended grid fits 32-bit indices
  const unsigned dummy = (unsigned)a.n_gproj;
  const unsigned long long empty = 0x0001000100010001ull * (unsigned long long)dummy;  // no ball in any layer
  double *sm = reinterpret_cast<double *>(dyn);
  double *ring = reinterpret_cast<double *>(dyn + col_planes_bytes(n, RY));
  const double *pcur = reinterpret_cast<const double *>(dyn + col_planes_bytes(n, RY) + col_ring_bytes(NS, RY));
  double *fb = slot<double>(a, 3);  // flush buffer: [layer][projector][plane][column]
  const double *veff = a.veff64;
  const unsigned long long *lid = a.lay_id;
  const double *lchi = a.lay_chi;
  const int NW = n * n2;     // window points (vector length)
  int *const st = a.status;  // (bounds-check build)
  (void)NW;
  (void)EV;
  (void)st;

  // zero the halo of the planes (the interior is written every plane)
  for (int i = tid; i < NPLANE * P2; i += NS) {
    const int r = (i % P2) / P, c = i % P;
    if (r < FDN || r >= n + FDN || c < FDN || c >= n + FDN) sm[i] = 0.0;
  }

  int y[RY], col[RY];
  bool ok[RY];
  int xb[RY];
#pragma unroll
  for (int j = 0; j < RY; j++) {
    y[j] = yb + j;
    ok[j] = tv && y[j] < n;
    col[j] = ok[j] ? y[j] * n + x : 0;
    xb[j] = (S.gk * a.ey + (S.gj + (ok[j] ? y[j] : 0))) * a.ex + S.gi + x;
  }
  // ring slot of (row j, plane zz): ring[((zz mod CRSLOT) * RY + j) * NS + tid]
  auto rslot = [&](int j, int zz) -> double & { return ring[(((zz + CRSLOT) & (CRSLOT - 1)) * RY + j) * NS + tid]; };

  // the stencil input of row j at plane zz (LZF: formed from the loaded operands)
  double fut[RY][F];
  double pf[RY], r1[RY], r2[RY];
  auto load_ops = [&](int j, int zz) {
    if (!ok[j] || zz >= n) return;
    const int g = SQB_IDX(zz * n2 + col[j], NW, st);
    pf[j] = io.vin[g];
    if constexpr (SK == SK_LZF) {
      r1[j] = io.p1[g];
      r2[j] = io.p2[g];
    }
  };
  auto next_in = [&](int j, int zz) -> double {
    if (!ok[j] || zz >= n) return 0.0;
    const int g = zz * n2 + col[j];
    double v;
    if constexpr (SK == SK_LZF) v = io.s1 * (pf[j] - io.ca * r1[j]) - io.cb * r2[j];
    else v = pf[j];
    if constexpr (SK == SK_LZF) io.wout[SQB_IDX(g, NW, st)] = v;
    (void)g;
    return v;
  };

  // per-plane point data, loaded one plane ahead
  double ve[RY];
  double q1[RY];
  unsigned long long idc[RY] = {}, idn[RY] = {};
  double acd[RY][KL][CPM];
  auto load_ids = [&](int j, int zz) -> unsigned long long {
    return (ok[j] && zz < n) ? __ldg(lid + SQB_IDX(xb[j] + zz * EP, EV, st)) : empty;
  };
  auto load_point = [&](int j, int zz) {
    if (!ok[j] || zz >= n) return;
    const int X = SQB_IDX(xb[j] + zz * EP, EV, st);
    if constexpr (STENCIL) ve[j] = __ldg(veff + X);
    if constexpr (SK == SK_CH) {
      if (!io.first) q1[j] = io.p1[SQB_IDX(zz * n2 + col[j], NW, st)];
    }
    (void)X;
  };
  auto chi_at = [&](int j, int k, int q, int X) -> double {
    return lay_of(idc[j], k) != dummy ? __ldg(lchi + (k * CPM + q) * EV + X) : 0.0;
  };

#pragma unroll
  for (int j = 0; j < RY; j++) {
    ve[j] = 0.0;
    q1[j] = 0.0;
#pragma unroll
    for (int k = 0; k < KL; k++) {
#pragma unroll
      for (int q = 0; q < CPM; q++) acd[j][k][q] = 0.0;
    }
    idc[j] = load_ids(j, 0);
    idn[j] = load_ids(j, 1);
    if constexpr (STENCIL) {
      // planes behind the window are zero; planes 0..FDN enter it
#pragma unroll
      for (int s = 1; s <= FDN; s++) rslot(j, -s) = 0.0;
#pragma unroll
      for (int s = 0; s <= FDN; s++) {
        load_ops(j, s);
        fut[j][s] = next_in(j, s);
      }
      load_ops(j, FDN + 1);
    }
    load_point(j, 0);
  }
  const double c0 = 3.0 * a.coeff_lap[0];
  const double rcb = SK == SK_CH ? 1.0 / io.cb : 0.0;

  // Planes through the shared buffers with the split barrier of sqb_sweep.cuh.
  const int sofs = (yb + FDN) * P + x + FDN;  // the thread's first row in a plane buffer
  if constexpr (STENCIL) {
#pragma unroll
    for (int j = 0; j < RY; j++)
      if (ok[j]) sm[sofs + j * P] = fut[j][0];
  }
  bar_sweep(NS);  // halo and plane 0 written; the previous sweep's phases are counted
  const unsigned ph0 = S.pbar_phase;
  int bz = 0;  // buffer of plane z
  for (int z = 0; z < n; z++) {
    double *smz = sm + bz * P2;
    const int bn = bz == NPLANE - 1 ? 0 : bz + 1;
    if constexpr (STENCIL) {
      if (z + 1 < n) {
#pragma unroll
        for (int j = 0; j < RY; j++)
          if (ok[j]) sm[bn * P2 + sofs + j * P] = fut[j][1];
        __syncwarp();
        if (lane == 0) pbar_arrive(&S.pbar);
      }
    }
    if (tv) {
      double hv[RY], v[RY];
      if constexpr (STENCIL) {
        // arm k of each point sums (x-k) + (x+k) + (y-k) + (y+k) + (z-k) + (z+k)
        // in that order before the coefficient, as HsubTimesVec does
        // (sq.cpp:894-897).  The RY rows y0..y0+RY-1 of a thread share their
        // y-arm loads: arm k loads rows y0-k and y0+RY-1+k; row j's y0+j-k is
        // the centre of row j-k when j >= k, and its y0+j+k the centre of row
        // j+k when j+k < RY.
        const double *cp0 = smz + (yb + FDN) * P + x + FDN;
        double temp[RY];
#pragma unroll
        for (int j = 0; j < RY; j++) temp[j] = fut[j][0] * c0;
        if constexpr (RY == 2) {
          // the loads of the previous arm carried in two registers
          const double *c1p = cp0 + P;
          double prev_m = fut[0][0], prev_p = fut[1][0];
#pragma unroll
          for (int k = 1; k <= FDN; k++) {
            const double ym = cp0[-k * P], yp = c1p[k * P];
            const double zm0 = rslot(0, z - k), zm1 = rslot(1, z - k);
            const double s0 = cp0[-k] + cp0[k] + ym + prev_p + zm0 + fut[0][k];
            const double s1 = c1p[-k] + c1p[k] + prev_m + yp + zm1 + fut[1][k];
            temp[0] += s0 * a.coeff_lap[k];
            temp[1] += s1 * a.coeff_lap[k];
            prev_m = ym;
            prev_p = yp;
          }
        } else {
          double ym[FDN + 1], yp[FDN + 1];
#pragma unroll
          for (int k = 1; k <= FDN; k++) {
            ym[k] = cp0[-k * P];
            yp[k] = cp0[(RY - 1 + k) * P];
#pragma unroll
            for (int j = 0; j < RY; j++) {
              const double *cj = cp0 + j * P;
              const double ylo = j >= k ? fut[j >= k ? j - k : 0][0] : ym[j >= k ? 1 : k - j];
              const double yhi = j + k < RY ? fut[j + k < RY ? j + k : 0][0] : yp[j + k < RY ? 1 : j + k - RY + 1];
              const double zm = rslot(j, z - k);
              const double sj = cj[-k] + cj[k] + ylo + yhi + zm + fut[j][k];
              temp[j] += sj * a.coeff_lap[k];
            }
          }
        }
#pragma unroll
        for (int j = 0; j < RY; j++) {
          const int X = xb[j] + z * EP;
          double vnl = 0.0;
#pragma unroll
          for (int k = 0; k < KL; k++) {
            const unsigned id = lay_of(idc[j], k);
#pragma unroll
            for (int q = 0; q < CPM; q++) vnl += pcur[SQB_IDX(id + q, a.n_gproj + CPM, st)] * chi_at(j, k, q, X);
          }
          v[j] = fut[j][0];
          hv[j] = -0.5 * temp[j] + ve[j] * v[j] + vnl;
        }
      }
#pragma unroll
      for (int j = 0; j < RY; j++) {
        if (!ok[j]) continue;
        const int g = SQB_IDX(z * n2 + col[j], NW, st);
        double o;
        if constexpr (SK == SK_ONES) {
          o = start_val(io.chk, g);
        } else if constexpr (SK == SK_LZF) {
          o = hv[j];
          io.out[g] = o;
          acc0 += v[j] * v[j];
          acc1 += v[j] * hv[j];
        } else {
          // sq.cpp:588, 615 divide by zee; the sweep multiplies by 1/zee
          // (one rounding apart, no FP64 division per point)
          if (io.first) o = (hv[j] - io.ca * v[j]) * rcb;
          else o = (2.0 * (hv[j] - io.ca * v[j])) * rcb - q1[j];
          io.out[g] = o;
          if (io.dbl) {
            acc0 += o * o;
            acc1 += o * v[j];
          }
        }
        if (g == gc) S.center_val = o;
        if (!isfinite(o)) atomicOr(a.status, ST_NONFINITE);
        const int X = xb[j] + z * EP;
#pragma unroll
        for (int k = 0; k < KL; k++) {
#pragma unroll
          for (int q = 0; q < CPM; q++) acd[j][k][q] += chi_at(j, k, q, X) * o;
        }
        // a column that leaves a layer's ball after plane z flushes its partial
        // to the slot of (layer, z, column)
        const unsigned long long chg = idc[j] ^ idn[j];
        if (z + 1 < n && chg != 0ull) {
#pragma unroll
          for (int k = 0; k < KL; k++) {
            if (lay_of(chg, k) == 0u) continue;
            if (lay_of(idc[j], k) != dummy) {
#pragma unroll
              for (int q = 0; q < CPM; q++)
                fb[SQB_IDX(((k * CPM + q) * n + z) * n2 + col[j], KL * CPM * NW, st)] = acd[j][k][q];
            }
#pragma unroll
            for (int q = 0; q < CPM; q++) acd[j][k][q] = 0.0;
          }
        }
      }
    }
    // advance: ids, point data and the stencil input
#pragma unroll
    for (int j = 0; j < RY; j++) {
      idc[j] = idn[j];
      idn[j] = load_ids(j, z + 2);
      load_point(j, z + 1);
      if constexpr (STENCIL) {
        rslot(j, z) = fut[j][0];  // plane z moves behind (its slot is free: CRSLOT > FDN)
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
  }
  if constexpr (STENCIL) {
    // every thread read ph0 before its warp's first arrival, and thread 0
    // passed every wait of this sweep
    if (tid == 0) S.pbar_phase = ph0 + (unsigned)(n - 1);
  }
  // balls that end at the window's last plane: every layer's open partial (a
  // layer with no ball there writes a zero no reduction reads); then every
  // ball's columns are summed
  if (tv) {
#pragma unroll
    for (int j = 0; j < RY; j++) {
      if (!ok[j]) continue;
#pragma unroll
      for (int k = 0; k < KL; k++) {
#pragma unroll
        for (int q = 0; q < CPM; q++)
          fb[SQB_IDX(((k * CPM + q) * n + n - 1) * n2 + col[j], KL * CPM * NW, st)] = acd[j][k][q];
      }
    }
  }
  bar_sweep(NS);
  for (int p = warp; p < S.n_pi; p += nwarp) col_reduce(a, S, fb, p, lane);
  bar_sweep(NS);
}

template <int RY>
struct ColumnTile {
  static constexpr int PM = CPM;
  static __device__ __forceinline__ int cols(int n) { return n; }
  static __device__ __forceinline__ int shift(const Shared &) { return 0; }
  template <typename T, int SK>
  static __device__ __forceinline__ void run(const SweepArgs &a, Shared &S, unsigned char *dyn, const IO<T> &io,
                                             double &acc0, double &acc1) {
    static_assert(std::is_same<T, double>::value && (SK == SK_ONES || SK == SK_LZF || SK == SK_CH), "FP64 SQ step only");
    col_sweep<SK, RY>(a, S, dyn, io, acc0, acc1);
  }
};

template <int MAXT, int RY>
__global__ void __launch_bounds__(MAXT, 1) sweep_cols_kernel(SweepArgs a) {
  using Tile = ColumnTile<RY>;
  extern __shared__ __align__(128) unsigned char smem[];
  Shared &S = *reinterpret_cast<Shared *>(smem);
  unsigned char *dyn = smem + shared_fixed();
  double *pcur = reinterpret_cast<double *>(dyn + col_planes_bytes(a.n, RY) + col_ring_bytes(a.nsweep, RY));
  for (int i = threadIdx.x; i < a.n_gproj + CPM; i += blockDim.x) pcur[i] = 0.0;  // [n_gproj..]: the empty id
  pbar_setup(S);
  for (;;) {
    if (threadIdx.x == 0) {
      const int q = atomicAdd(a.counter, 1);
      S.qidx = q;
      S.node = q < (a.n_list_dev ? *a.n_list_dev : a.n_list) ? a.node_list[q] : -1;
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
    lanczos<Tile, double, false>(a, S, dyn, pcur, lmin, lmax, rows);
    const double chi = (lmax + lmin) / 2, zee = (lmax - lmin) / 2;  // sq.cpp:564-565
    count_proj_points(a, S, rows + 1, 0);
    moments<Tile>(a, S, dyn, pcur, chi, zee, a.rho_pj + (size_t)node * (a.npl + 1));
    count_proj_points(a, S, a.npl / 2, 1);
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

// Launch bounds, which set the registers per thread: windows up to 31 wide run
// 512 threads (128 registers), 33 wide 576 (96), up to 43 wide 1024 (64); three
// rows per thread, up to 33 wide, 384 (168).
constexpr int COL_A = 512, COL_B = 576, COL_C = 1024, COL_R3 = 384;
const void *cols_kernel(int n, int ry) {
  const int t = col_threads(n, ry);
  if (ry == 3) return t <= COL_R3 ? reinterpret_cast<const void *>(&sweep_cols_kernel<COL_R3, 3>) : nullptr;
  if (ry != 2) return nullptr;
  return t <= COL_A   ? reinterpret_cast<const void *>(&sweep_cols_kernel<COL_A, 2>)
         : t <= COL_B ? reinterpret_cast<const void *>(&sweep_cols_kernel<COL_B, 2>)
         : t <= COL_C ? reinterpret_cast<const void *>(&sweep_cols_kernel<COL_C, 2>)
                      : nullptr;
}

size_t cols_smem(int n, int n_gproj, int ry) {
  return shared_fixed() + col_planes_bytes(n, ry) + col_ring_bytes(col_threads(n, ry), ry) +
         (((size_t)(n_gproj + CPM) * sizeof(double) + 127) & ~size_t(127));
}

}  // namespace

bool sweep_cols_supported(int n, int n_gproj, int ry, size_t smem_limit) {
  return cols_kernel(n, ry) != nullptr && cols_smem(n, n_gproj, ry) <= smem_limit;
}

int sweep_cols_threads(int n, int ry) { return col_threads(n, ry); }

cudaError_t sweep_cols_per_sm(const SweepArgs &a, int *per_sm) {
  if (col_threads(a.n, a.ry) != a.nsweep || a.pmax != CPM || a.form != 0) return cudaErrorInvalidConfiguration;
  return kernel_setup(cols_kernel(a.n, a.ry), a.nsweep, cols_smem(a.n, a.n_gproj, a.ry), per_sm);
}

cudaError_t launch_sweep_cols(const SweepArgs &a, int grid, cudaStream_t s) {
  cudaError_t e = sweep_cols_per_sm(a, nullptr);
  if (e != cudaSuccess) return e;
  SweepArgs args = a;
  void *argv[] = {&args};
  return cudaLaunchKernel(cols_kernel(a.n, a.ry), dim3(grid), dim3(a.nsweep), argv, cols_smem(a.n, a.n_gproj, a.ry), s);
}

}  // namespace sqb

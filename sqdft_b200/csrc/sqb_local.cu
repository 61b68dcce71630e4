// Pseudocharge density and local forces on the device: the per-atom loops of
// ChargeDensity (initialize.cpp:470-784) and ForcesLocal (forces.cpp:20-315).
//
// Every atom replica J whose rb-box meets the block contributes, on its
// intersection box, b_J = -(1/4 pi) Lap_h V_J and the same of the smooth
// reference potential V~_J, with V_J the spline of r Vloc over r.
//
// Charge density: one CTA per 8^3 tile of the block, two threads per node (one
// for V_J, one for V~_J: the tile's 128 KB of shared memory leave room for one
// CTA per SM, and its 32 warps hide the lookups' latency where 16 did not).
// The CTA lists the replicas that meet its tile, in the reference's loop
// order, and for each one puts V_J and V~_J on the tile and its FDN halo
// into shared memory. Each thread then adds the replica's terms to its own
// node. A node therefore sums its replicas in the reference's order, and its
// b and rho_at equal the reference's bit for bit. This translation unit is
// compiled without multiply-add contraction, as the reference's x86 build
// runs.
//
// Local forces: each replica's V_J, V~_J (box + 2 FDN) and b_J, b~_J
// (box + FDN) go into a scratch box in global memory. The contraction over
// the box is spread over LOC_FORCE_CTAS CTAs per replica, with a fixed
// reduction order.
#include "sqb_internal.cuh"

namespace sqb {

namespace {

constexpr int LT = LOC_TILE;
constexpr int LH = LT + 2 * FDN;  // halo'd tile edge
constexpr int LH3 = LH * LH * LH;
constexpr int LLIST = 512;        // replicas tested per list pass (one per thread)
constexpr double PI = 3.14159265358979323846;  // M_PI
constexpr double TOL = 1e-12;                  // TEMP_TOL of the reference

// A type's prepared radial tables (launch_local_prepare): per interval the
// cubic's coefficients of rVloc and of the atomic density, as ispline_gen
// forms them at each point, and per bin of the radius the first grid point at
// or above the bin's lower edge.  A bin is the exponent and the top six
// mantissa bits of the radius (1/64 of an octave), so a lookup searches the one
// or two grid points of its bin and not the whole grid: three dependent loads
// in place of the binary search's eleven and no division.
constexpr int BIN0 = (1023 - 12) << 6;  // bins start at 2^-12 and end at 2^9
constexpr int NBIN = 21 << 6;
__device__ __forceinline__ int radius_bin(double x) {
  const int b = (__double2hiint(x) >> 14) - BIN0;
  return b < 0 ? 0 : (b >= NBIN ? NBIN - 1 : b);
}

// First grid point >= x among [lo, hi].
__device__ __forceinline__ int first_at_or_above(const double *X, int lo, int hi, double x) {
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (X[mid] < x) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

__global__ void local_prepare_kernel(const double *tab, const long long *off, const int *size, double4 *coef, int *bin) {
  const int t = blockIdx.y, len = size[t];
  const double *X = tab + off[t];
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < 2 * len + NBIN + 1; i += gridDim.x * blockDim.x) {
    if (i < 2 * len) {
      const int f = i >= len, j = i - f * len;
      if (j > len - 2) continue;
      const double *Y = X + (f ? 3 : 1) * (size_t)len, *YD = Y + len;
      const double dx = 1.0 / (X[j + 1] - X[j]);
      const double dy = (Y[j + 1] - Y[j]) * dx;
      const double A2 = dx * (3.0 * dy - 2.0 * YD[j] - YD[j + 1]);
      const double A3 = dx * dx * (-2.0 * dy + YD[j] + YD[j + 1]);
      coef[2 * (off[t] / 5) + i] = make_double4(Y[j], YD[j], A2, A3);
    } else {
      const int k = i - 2 * len;
      const double edge = __hiloint2double((k + BIN0) << 14, 0);
      bin[t * (NBIN + 1) + k] = k == 0 ? 0 : (k == NBIN ? len - 1 : first_at_or_above(X, 0, len - 1, edge));
    }
  }
}

// ispline_gen (spline.cpp:11-55) at one point: the interval below the first
// grid point >= x, stepped back unless equal (false out of the table's range),
// and the cubic of field f (0 rVloc, 1 the atomic density) there.
__device__ __forceinline__ bool spline_interval(const LocalArgs &a, int t, double x, int &j) {
  const double *X = a.tab + a.typ_off[t];
  const int len = a.typ_size[t];
  if (!(x >= X[0] && x <= X[len - 1])) return false;
  const int *bin = a.bin + t * (NBIN + 1) + radius_bin(x);
  j = first_at_or_above(X, bin[0], bin[1], x);
  if (x < X[j]) j--;
  if (j > len - 2) j = len - 2;
  if (j < 0) j = 0;
  return true;
}
__device__ __forceinline__ double spline_value(const LocalArgs &a, int t, int f, int j, double x) {
  const double *X = a.tab + a.typ_off[t];
  const double2 *c = reinterpret_cast<const double2 *>(a.coef + 2 * (a.typ_off[t] / 5) + (size_t)f * a.typ_size[t] + j);
  const double2 lo = c[0], hi = c[1];
  const double u = x - X[j];
  return ((hi.y * u + hi.x) * u + lo.y) * u + lo.x;
}

// Distance of global node (gi, gj, gk) from a replica (initialize.cpp:571).
__device__ __forceinline__ double node_radius(const LocalArgs &a, const double *c, int gi, int gj, int gk) {
  const double dx = gi * a.delta - c[0], dy = gj * a.delta - c[1], dz = gk * a.delta - c[2];
  return sqrt(dx * dx + dy * dy + dz * dz);
}

// VlocJ and VlocJ_tilda of a replica of type t at distance r
// (initialize.cpp:573-597, forces.cpp:126-143).
__device__ bool vloc_pair(const LocalArgs &a, int t, double r, double &v, double &vt) {
  int j;
  if (!spline_interval(a, t, r, j)) return false;
  const double s = spline_value(a, t, 0, j, r);
  if (fabs(r - 0.0) < TOL) {
    const double *G = a.tab + a.typ_off[t];
    v = G[a.typ_size[t] + 1] / G[1];
  } else {
    v = s / r;
  }
  const double rc = a.rc_tilda, Z = a.Z[t];
  if (r < rc)
    vt = -Z * (9 * pow(r, 7) - 30 * rc * pow(r, 6) + 28 * rc * rc * pow(r, 5) - 14 * pow(rc, 5) * pow(r, 2) +
               12 * pow(rc, 7)) /
         (5 * pow(rc, 8));
  else
    vt = -Z / r;
  return true;
}

// -(1/4 pi) Lap_h f at index q of a box with x stride 1, y stride sy and z
// stride sz (the expression of initialize.cpp:604-614, forces.cpp:154-170).
__device__ __forceinline__ double neg_lap(const LocalArgs &a, const double *f, long long q, long long sy, long long sz) {
  double s = f[q] * 3 * a.coeff_lap[0] * (-1 / (4 * PI));
#pragma unroll
  for (int k = 1; k <= FDN; k++)
    s += (f[q - k] + f[q + k] + f[q - k * sy] + f[q + k * sy] + f[q - k * sz] + f[q + k * sz]) * a.coeff_lap[k] *
         (-1 / (4 * PI));
  return s;
}

__device__ __forceinline__ double block_sum(double v, double *red) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) red[w] = v;
  __syncthreads();
  double s = 0.0;
  if (threadIdx.x == 0)
    for (int i = 0; i < (int)(blockDim.x >> 5); i++) s += red[i];
  return s;  // valid in thread 0
}

__global__ void __launch_bounds__(2 * LT *LT *LT) charge_density_kernel(LocalArgs a) {
  extern __shared__ double sm[];
  double *sV = sm, *sVt = sm + LH3;
  __shared__ int list[LLIST];
  __shared__ int wcount[2 * LT * LT * LT / 32 + 1];
  __shared__ int nlist;
  __shared__ double red[32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarp = blockDim.x >> 5;
  const int NX = a.np[0], NY = a.np[1], NZ = a.np[2];
  const int x0 = blockIdx.x * LT, y0 = blockIdx.y * LT, z0 = blockIdx.z * LT;  // tile origin (block nodes)
  const int half = tid / (LT * LT * LT);  // 0: V_J and the atomic density, 1: V~_J and Vc
  const int li = tid % LT, lj = (tid / LT) % LT, lk = tid / (LT * LT) % LT;
  const int x = x0 + li, y = y0 + lj, z = z0 + lk;
  const bool in = x < NX && y < NY && z < NZ;
  const int gx = x + a.pnode_s[0], gy = y + a.pnode_s[1], gz = z + a.pnode_s[2];
  // the tile's global node range (clipped to the block)
  const int tx0 = x0 + a.pnode_s[0], ty0 = y0 + a.pnode_s[1], tz0 = z0 + a.pnode_s[2];
  const int tx1 = min(x0 + LT, NX) - 1 + a.pnode_s[0], ty1 = min(y0 + LT, NY) - 1 + a.pnode_s[1],
            tz1 = min(z0 + LT, NZ) - 1 + a.pnode_s[2];
  const double h = a.delta;
  double b = 0.0, vc = 0.0, ra = 0.0;       // b of the thread's field; Vc (half 1), rho_at (half 0)
  double eS = 0.0, nC = 0.0, nE = 0.0;
  for (int base = 0; base < a.n_rep; base += LLIST) {
    // the replicas of [base, base + LLIST) whose box meets the tile, in order
    const int r = base + tid;
    bool hit = false;
    if (tid < LLIST && r < a.n_rep) {
      const int *bx = a.rep_box + 6 * r;
      hit = bx[0] <= tx1 && bx[1] >= tx0 && bx[2] <= ty1 && bx[3] >= ty0 && bx[4] <= tz1 && bx[5] >= tz0;
    }
    const unsigned bal = __ballot_sync(0xffffffffu, hit);
    if (lane == 0) wcount[warp] = __popc(bal);
    __syncthreads();
    if (tid == 0) {
      int s = 0;
      for (int w = 0; w < nwarp; w++) {
        const int c = wcount[w];
        wcount[w] = s;
        s += c;
      }
      nlist = s;
    }
    __syncthreads();
    if (hit) list[wcount[warp] + __popc(bal & ((1u << lane) - 1u))] = r;
    __syncthreads();
    const int nl = nlist;
    for (int q = 0; q < nl; q++) {
      const int rr = list[q], t = a.rep_type[rr];
      const int *bx = a.rep_box + 6 * rr;
      const double *c = a.rep_xyz + 3 * rr;
      // V and V~ on the halo'd tile where the replica's box + FDN covers it
      for (int p = tid; p < LH3; p += blockDim.x) {
        const int Gx = tx0 - FDN + p % LH, Gy = ty0 - FDN + (p / LH) % LH, Gz = tz0 - FDN + p / (LH * LH);
        if (Gx >= bx[0] - FDN && Gx <= bx[1] + FDN && Gy >= bx[2] - FDN && Gy <= bx[3] + FDN && Gz >= bx[4] - FDN &&
            Gz <= bx[5] + FDN) {
          double v, vt;
          if (!vloc_pair(a, t, node_radius(a, c, Gx, Gy, Gz), v, vt)) {
            atomicOr(a.status, ST_SPLINE_RANGE);
            v = vt = 0.0;
          }
          sV[p] = v;
          sVt[p] = vt;
        }
      }
      __syncthreads();
      if (in && gx >= bx[0] && gx <= bx[1] && gy >= bx[2] && gy <= bx[3] && gz >= bx[4] && gz <= bx[5]) {
        const long long hc = ((long long)(lk + FDN) * LH + (lj + FDN)) * LH + (li + FDN);
        // initialize.cpp:583-588: the atomic density at the node
        if (!half) {
          const double r = node_radius(a, c, gx, gy, gz);
          double rho_temp = 0.0;
          int j;
          if (spline_interval(a, t, r, j)) rho_temp = spline_value(a, t, 1, j, r);
          else atomicOr(a.status, ST_SPLINE_RANGE);
          ra += rho_temp;
          nE += rho_temp * h * h * h;
        }
        // initialize.cpp:600-626
        const double *f = half ? sVt : sV;
        const double bJ = neg_lap(a, f, hc, LH, LH * LH);
        b += bJ;
        eS += 0.5 * bJ * f[hc] * h * h * h;
        nC += bJ * h * h * h;
        if (half) vc += sVt[hc] - sV[hc];
      }
      __syncthreads();
    }
  }
  if (in) {
    const long long g = ((long long)z * NY + y) * NX + x;
    if (half) {
      a.b_tilda[g] = b;
      a.vc[g] = vc;
    } else {
      a.b[g] = b;
      a.rho_at[g] = ra;
    }
  }
  const int nb = gridDim.x * gridDim.y * gridDim.z, blk = (blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
  // (the other half's zeros leave each sum as it is)
  const double sums[5] = {half ? 0.0 : eS, half ? 0.0 : nC, nE, half ? nC : 0.0, half ? eS : 0.0};
  for (int k = 0; k < 5; k++) {
    const double s = block_sum(sums[k], red);
    if (tid == 0) a.partial[k * nb + blk] = s;
  }
}

__global__ void charge_finish_kernel(LocalArgs a, double scale, double shift) {
  __shared__ double red[32];
  const long long n = (long long)a.np[0] * a.np[1] * a.np[2];
  double e = 0.0;
  for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < n; g += (long long)gridDim.x * blockDim.x) {
    const double bt = scale * a.b_tilda[g];
    a.b_tilda[g] = bt;
    const double v = a.vc[g] + shift;
    a.vc[g] = v;
    e += 0.5 * (bt + a.b[g]) * v * a.h3;
  }
  const double s = block_sum(e, red);
  if (threadIdx.x == 0) a.partial[blockIdx.x] = s;
}

// Scratch box of replica r: extent box + 2 FDN per side.
struct SBox {
  int nx, ny, nz, i0, j0, k0;
};
__device__ __forceinline__ SBox sbox(const LocalArgs &a, int r) {
  const int *bx = a.rep_box + 6 * r;
  SBox s;
  s.nx = bx[1] - bx[0] + 1 + 4 * FDN;
  s.ny = bx[3] - bx[2] + 1 + 4 * FDN;
  s.nz = bx[5] - bx[4] + 1 + 4 * FDN;
  s.i0 = bx[0] - 2 * FDN;
  s.j0 = bx[2] - 2 * FDN;
  s.k0 = bx[4] - 2 * FDN;
  return s;
}

// forces.cpp:116-143: VlocJ, VlocJ_tilda on the box + 2 FDN.
__global__ void local_v_kernel(LocalArgs a, int r0) {
  const int r = r0 + blockIdx.y, t = a.rep_type[r];
  const SBox s = sbox(a, r);
  const long long nb = (long long)s.nx * s.ny * s.nz;
  double *V = a.scr + a.scr_off[r], *Vt = V + nb;
  const double *c = a.rep_xyz + 3 * r;
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < nb; p += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(p % s.nx), j = (int)((p / s.nx) % s.ny), k = (int)(p / ((long long)s.nx * s.ny));
    double v, vt;
    if (!vloc_pair(a, t, node_radius(a, c, s.i0 + i, s.j0 + j, s.k0 + k), v, vt)) {
      atomicOr(a.status, ST_SPLINE_RANGE);
      v = vt = 0.0;
    }
    V[p] = v;
    Vt[p] = vt;
  }
}

// forces.cpp:149-173: bJ, bJ_tilda on the box + FDN.
__global__ void local_b_kernel(LocalArgs a, int r0) {
  const int r = r0 + blockIdx.y;
  const SBox s = sbox(a, r);
  const long long nb = (long long)s.nx * s.ny * s.nz, sy = s.nx, sz = (long long)s.nx * s.ny;
  double *V = a.scr + a.scr_off[r], *Vt = V + nb, *bJ = Vt + nb, *bJt = bJ + nb;
  const int mx = s.nx - 2 * FDN, my = s.ny - 2 * FDN, mz = s.nz - 2 * FDN;
  const long long m = (long long)mx * my * mz;
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < m; p += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(p % mx) + FDN, j = (int)((p / mx) % my) + FDN, k = (int)(p / ((long long)mx * my)) + FDN;
    const long long q = ((long long)k * s.ny + j) * s.nx + i;
    bJ[q] = neg_lap(a, V, q, sy, sz);
    bJt[q] = neg_lap(a, Vt, q, sy, sz);
  }
}

// forces.cpp:178-277: the gradients along x, y, z of bJ, bJ_tilda, VlocJ and
// VlocJ_tilda on the intersection box and the local and correction force
// terms; per-CTA sums into fpart.
__global__ void local_force_kernel(LocalArgs a, int r0) {
  __shared__ double red[32];
  const int r = r0 + blockIdx.y;
  const SBox s = sbox(a, r);
  const long long nb = (long long)s.nx * s.ny * s.nz;
  const long long st[3] = {1, s.nx, (long long)s.nx * s.ny};
  const double *V = a.scr + a.scr_off[r], *Vt = V + nb, *bJ = Vt + nb, *bJt = bJ + nb;
  const int NX = a.np[0], NY = a.np[1], PX = NX + 2 * FDN, PY = NY + 2 * FDN;
  const int mx = s.nx - 4 * FDN, my = s.ny - 4 * FDN, mz = s.nz - 4 * FDN;
  const long long m = (long long)mx * my * mz;
  double fl[3] = {0, 0, 0}, fc[3] = {0, 0, 0};
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < m; p += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(p % mx) + 2 * FDN, j = (int)((p / mx) % my) + 2 * FDN,
              k = (int)(p / ((long long)mx * my)) + 2 * FDN;
    const long long q = ((long long)k * s.ny + j) * s.nx + i;
    const int li = i + s.i0 - a.pnode_s[0], lj = j + s.j0 - a.pnode_s[1], lk = k + s.k0 - a.pnode_s[2];
    const double ph = a.phi[((long long)(lk + FDN) * PY + (lj + FDN)) * PX + (li + FDN)];
    const long long g = ((long long)lk * NY + lj) * NX + li;
    const double vcg = a.vcf[g], bsum = a.btf[g] + a.bf[g];
#pragma unroll
    for (int d = 0; d < 3; d++) {
      const long long sd = st[d];
      double Db = 0, Dbt = 0, DV = 0, DVt = 0;
#pragma unroll
      for (int k2 = 1; k2 <= FDN; k2++) Db += (-bJ[q - k2 * sd] + bJ[q + k2 * sd]) * a.coeff_grad[k2];
      fl[d] += Db * (ph - V[q]) * a.h3;
#pragma unroll
      for (int k2 = 1; k2 <= FDN; k2++) Dbt += (-bJt[q - k2 * sd] + bJt[q + k2 * sd]) * a.coeff_grad[k2];
#pragma unroll
      for (int k2 = 1; k2 <= FDN; k2++) DV += (-V[q - k2 * sd] + V[q + k2 * sd]) * a.coeff_grad[k2];
#pragma unroll
      for (int k2 = 1; k2 <= FDN; k2++) DVt += (-Vt[q - k2 * sd] + Vt[q + k2 * sd]) * a.coeff_grad[k2];
      fc[d] += 0.5 * (Dbt * (vcg - Vt[q]) + Db * (vcg + V[q]) + (DVt - DV) * bsum + bJ[q] * DV - bJt[q] * DVt) * a.h3;
    }
  }
  double *out = a.fpart + ((long long)blockIdx.y * gridDim.x + blockIdx.x) * 6;
  for (int d = 0; d < 3; d++) {
    const double s1 = block_sum(fl[d], red);
    if (threadIdx.x == 0) out[d] = s1;
    const double s2 = block_sum(fc[d], red);
    if (threadIdx.x == 0) out[3 + d] = s2;
  }
}

}  // namespace

size_t local_coef_count(long long table_values) { return (size_t)(2 * (table_values / 5)); }
size_t local_bin_count(int n_typ) { return (size_t)n_typ * (NBIN + 1); }

cudaError_t launch_local_prepare(int n_typ, const double *tab, const long long *off, const int *size, double4 *coef,
                                 int *bin, cudaStream_t s) {
  local_prepare_kernel<<<dim3(16, n_typ), 256, 0, s>>>(tab, off, size, coef, bin);
  return cudaGetLastError();
}

int charge_density_ctas(const int np[3]) {
  return ((np[0] + LT - 1) / LT) * ((np[1] + LT - 1) / LT) * ((np[2] + LT - 1) / LT);
}

cudaError_t launch_charge_density(const LocalArgs &a, cudaStream_t s) {
  const size_t smem = 2 * (size_t)LH3 * sizeof(double);
  cudaError_t e = cudaFuncSetAttribute(charge_density_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  const dim3 grid((a.np[0] + LT - 1) / LT, (a.np[1] + LT - 1) / LT, (a.np[2] + LT - 1) / LT);
  charge_density_kernel<<<grid, 2 * LT * LT * LT, smem, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_charge_finish(const LocalArgs &a, double scale, double shift, cudaStream_t s) {
  charge_finish_kernel<<<charge_density_ctas(a.np), 256, 0, s>>>(a, scale, shift);
  return cudaGetLastError();
}

cudaError_t launch_forces_local(const LocalArgs &a, int r0, int r1, cudaStream_t s) {
  if (r1 <= r0) return cudaSuccess;
  const dim3 grid(LOC_FORCE_CTAS, r1 - r0);
  local_v_kernel<<<grid, 256, 0, s>>>(a, r0);
  local_b_kernel<<<grid, 256, 0, s>>>(a, r0);
  local_force_kernel<<<grid, 256, 0, s>>>(a, r0);
  return cudaGetLastError();
}

}  // namespace sqb

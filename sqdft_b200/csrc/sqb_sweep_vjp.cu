// Adjoint of the Chebyshev moments on the sweep kernel's machinery, in its own
// translation unit so its register allocation is its own.
//
// L = sum_j g_j mu_j with mu_j = e_c^T T_j(Ht) e_c / h^3, Ht = (H - chi)/zee and
// the bounds held fixed.  The recursion's vectors t_k = T_k(Ht) e_c carry the
// whole gradient: with U_m = 2 (T_m + T_m-2 + ...) (the last term once for T_0)
// the adjoint vectors are a_k+1 = sum_j>k (g_j/h^3) U_j-1-k(Ht) e_c, so
//   dL/dHt = sum_k,l w_k w_l S_k+l+1 t_k t_l^T,   k + l < npl,
//   S_m = sum of g_j/h^3 over j = m, m + 2, ... <= npl,   w_0 = 1, w_k = 2,
// a Hankel quadratic form of the stored t_k:
//   dL/dVeff(x) = sum_k,l w_k w_l S_k+l+1 t_k(x) t_l(x) / zee, and with
//   dVnl/dR = sum_q (dchi_q chi_q^T + chi_q dchi_q^T) / Denom_q,
//   dL/dR = sum_q dchi_q . (sum_l C_ql t_l) / zee,
//   C_ql = 2 w_l / Denom_q sum_k w_k S_k+l+1 (chi_q . t_k).
// So one forward run of npl - 1 sweeps whose vectors are kept (npl window
// vectors per CTA), and no reverse recursion: three times fewer matvecs than
// checkpoints with recomputation and a reverse Clenshaw recursion, for about
// npl^2 / 4 multiply-adds per window point, which stay in registers.
#include "sqb_sweep.cuh"

namespace sqb {

namespace {

using namespace sweep;

constexpr int VB = 16, VL = 8;  // vectors of a block of the quadratic form, and loaded at a time

// S_m of the node, m < vjp_weights(npl), zero beyond npl.
__host__ __device__ constexpr int vjp_weights(int npl) { return 2 * npl + 2 * VB + 2; }

template <int PM, int RY, int NT>
__device__ void node_vjp(const SweepArgs &a, Shared &S, unsigned char *dyn, double *pcur, double chi, double zee,
                         const double *g) {
  const int n = a.n, nl = a.nloc, npl = a.npl, NP = pair_cols(n), HX = NP >> 1, VP = n * NP, NW = n * VP;
  const int sh = S.gi & 1, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarp = blockDim.x >> 5;
  double *T = a.vjp + (size_t)blockIdx.x * a.vjp_stride;  // [npl][NW]
  double *Pk = T + (size_t)npl * NW;                       // [MAXP][npl]: chi . t_k
  double *Cl = Pk + (size_t)MAXP * npl;                    // [MAXP][npl]
  double *Sg = Cl + (size_t)MAXP * npl;                    // [vjp_weights]
  double d0 = 0.0, d1 = 0.0;
  if (tid == 0) {  // t_0 = e_c (its vector is zero elsewhere)
    const int c = (nl * n + nl) * NP + nl;
    T[c + sh] = 1.0;
    T[c + 1 - sh] = 0.0;
  }
  centre_projections(a, S, pcur);
  for (int p = tid; p < S.n_pi; p += blockDim.x) Pk[(size_t)p * npl] = S.pw_cur[p];
  for (int k = 1; k < npl; k++) {  // t_k = 2 Ht t_k-1 - t_k-2 (t_1 = Ht t_0)
    IO<double> io;
    io.vin = T + (size_t)(k - 1) * NW;
    io.p1 = k > 1 ? T + (size_t)(k - 2) * NW : io.vin;
    io.first = k == 1;
    io.out = T + (size_t)k * NW;
    io.ca = chi;
    io.cb = zee;
    sweep::sweep<double, PM, SK_CH, RY, NT>(a, S, dyn, io, d0, d1);
    for (int p = tid; p < S.n_pi; p += blockDim.x) Pk[(size_t)p * npl + k] = S.p_nxt[p];
    rotate(S, pcur);
  }
  // the weights, in the (now free) ring where they fit
  const int nS = vjp_weights(npl);
  double *Sw = (size_t)nS * sizeof(double) <= ring_bytes(NT, RY)
                   ? reinterpret_cast<double *>(dyn + planes_bytes(n, RY))
                   : Sg;
  for (int m = tid; m < nS; m += blockDim.x) {
    double s = 0.0;
    for (int j = npl - ((npl - m) & 1); j >= m && j >= 1; j -= 2) s += g[j] / a.h3;
    Sw[m] = m >= 1 && m <= npl ? s : 0.0;
  }
  __syncthreads();
  const double iz = 1.0 / zee;
  const bool at = a.g_atoms != nullptr;
  double *uf = slot<double>(a, 3);  // (the flush buffer) [layer][q][NW]: sum_l C_ql t_l at each point of a ball
  if (at) {
    // C_ql / w_l, and the balls' first local instances by global projector id
    for (int i = tid; i < S.n_pi * npl; i += blockDim.x) {
      const int p = i / npl, l = i - p * npl;
      const double *pk = Pk + (size_t)p * npl;
      double s = Sw[l + 1] * pk[0];
      for (int k = 1; k + l < npl; k++) s += 2.0 * Sw[k + l + 1] * pk[k];
      Cl[i] = 2.0 * s / S.p_den[p];
    }
    for (int p = tid; p < S.n_pi; p += blockDim.x) *reinterpret_cast<int *>(pcur + S.pi_g[p]) = p;
    __syncthreads();
  }
  // A pair of columns per thread: blocks K <= L of the weighted vectors w_k t_k,
  // K in registers, so each block pair loads its values once per point and does
  // VB^2 multiply-adds on them; the first K passes all vectors and forms the
  // atoms' sums on the way, so the vectors (1.5 GB at 27^3 windows and npl 64)
  // are not read again for each ball.
  const unsigned dummy = (unsigned)a.n_gproj;
  // (a ball with fewer than PM projectors reads on into the next one's Cl, or
  // past the last into the weights; nothing reads those sums)
  const int nC = MAXP * npl + vjp_weights(npl);
  const long long nV = a.evol / a.ex * a.gex;  // values of g_veff
  (void)nC;
  (void)nV;
  for (int i = tid; i < NW / 2; i += blockDim.x) {
    const int row = i / HX, x = 2 * (i - row * HX) - sh, z = row / n, y = row - z * n;
    const double *tp = T + 2 * i;
    const long long nT = (long long)npl * NW;
    (void)nT;
    const bool in0 = x >= 0, in1 = x + 1 < n;
    int off[KL][2];
    double2 u[KL][PM];
    if (at) {
      const ulonglong2 id = __ldg(reinterpret_cast<const ulonglong2 *>(
          a.lay_id + SQB_IDX(((S.gk + z) * a.ey + S.gj + y) * a.ex + S.gi + x, a.evol - 1, a.status)));
#pragma unroll
      for (int k = 0; k < KL; k++) {
        const unsigned i0 = lay_of(id.x, k), i1 = lay_of(id.y, k);
        off[k][0] = in0 && i0 != dummy ? *reinterpret_cast<const int *>(pcur + SQB_IDX(i0, a.n_gproj, a.status)) * npl : -1;
        off[k][1] = in1 && i1 != dummy ? *reinterpret_cast<const int *>(pcur + SQB_IDX(i1, a.n_gproj, a.status)) * npl : -1;
#pragma unroll
        for (int q = 0; q < PM; q++) u[k][q] = make_double2(0.0, 0.0);
      }
    }
    auto atoms = [&](int l, const double2 &t) {
#pragma unroll
      for (int k = 0; k < KL; k++) {
#pragma unroll
        for (int q = 0; q < PM; q++) {
          if (off[k][0] >= 0) u[k][q].x += Cl[SQB_IDX(off[k][0] + q * npl + l, nC, a.status)] * t.x;
          if (off[k][1] >= 0) u[k][q].y += Cl[SQB_IDX(off[k][1] + q * npl + l, nC, a.status)] * t.y;
        }
      }
    };
    double gx = 0.0, gy = 0.0;
    for (int K0 = 0; 2 * K0 < npl; K0 += VB) {
      double2 tk[VB];
#pragma unroll
      for (int k = 0; k < VB; k++)
        tk[k] = K0 + k < npl ? __ldcg(reinterpret_cast<const double2 *>(tp + SQB_IDX((size_t)(K0 + k) * NW, nT - 2 * i - 1, a.status))) : make_double2(0.0, 0.0);
#pragma unroll
      for (int k = 0; k < VB; k++) {
        const double w = K0 + k ? 2.0 : 1.0;
        tk[k].x *= w;
        tk[k].y *= w;
      }
      if (at && K0 == 0) {
#pragma unroll
        for (int k = 0; k < VB; k++)
          if (k < npl) atoms(k, tk[k]);
      }
      // the block with itself
#pragma unroll
      for (int l = 0; l < VB; l++) {
        double cx = 0.0, cy = 0.0;
#pragma unroll
        for (int k = 0; k < l; k++) {
          const double s = Sw[2 * K0 + k + l + 1];
          cx += s * tk[k].x;
          cy += s * tk[k].y;
        }
        const double s = Sw[SQB_IDX(2 * K0 + 2 * l + 1, nS, a.status)];
        gx += tk[l].x * (2.0 * cx + s * tk[l].x);
        gy += tk[l].y * (2.0 * cy + s * tk[l].y);
      }
      // with the later blocks, VL vectors at a time
      for (int L0 = K0 + VB; K0 + L0 < npl; L0 += VL) {
        double2 tl[VL];
#pragma unroll
        for (int l = 0; l < VL; l++)
          tl[l] = L0 + l < npl ? __ldcg(reinterpret_cast<const double2 *>(tp + SQB_IDX((size_t)(L0 + l) * NW, nT - 2 * i - 1, a.status))) : make_double2(0.0, 0.0);
#pragma unroll
        for (int l = 0; l < VL; l++) {
          tl[l].x *= 2.0;
          tl[l].y *= 2.0;
          const double *s = Sw + SQB_IDX(K0 + L0 + l + 1, nS - VB + 1, a.status);
          double cx = 0.0, cy = 0.0;
#pragma unroll
          for (int k = 0; k < VB; k++) {
            const double sk = s[k];
            cx += sk * tk[k].x;
            cy += sk * tk[k].y;
          }
          gx += 2.0 * tl[l].x * cx;  // both orders of the pair
          gy += 2.0 * tl[l].y * cy;
          if (at && K0 == 0 && L0 + l < npl) atoms(L0 + l, tl[l]);
        }
      }
    }
    // the window of node (gi, gj, gk) starts there in the halo'd block
    const long long v0 = ((long long)(S.gk + z) * a.ey + (S.gj + y)) * a.gex + (S.gi + x);
    if (in0) atomicAdd(a.g_veff + SQB_IDX(v0, nV, a.status), gx * iz);
    if (in1) atomicAdd(a.g_veff + SQB_IDX(v0 + 1, nV, a.status), gy * iz);
    if (at) {
#pragma unroll
      for (int k = 0; k < KL; k++)
#pragma unroll
        for (int q = 0; q < PM; q++)
          *reinterpret_cast<double2 *>(uf + SQB_IDX((size_t)(k * PM + q) * NW + 2 * i, (size_t)KL * PM * NW - 1, a.status)) =
              u[k][q];
    }
  }
  if (!at) return;
  __syncthreads();
  // dL/dR: a warp per replica ball
  for (int p = tid; p < S.n_pi; p += blockDim.x) pcur[S.pi_g[p]] = 0.0;
  for (int e = warp; e < S.n_ent; e += nwarp) {
    const int x0 = S.e_x0[e], y0 = S.e_y0[e], z0 = S.e_z0[e];
    const int bx = S.e_x1[e] - x0 + 1, by = S.e_y1[e] - y0 + 1, vol = bx * by * (S.e_z1[e] - z0 + 1);
    const int r = S.e_r[e], np = S.e_np[e], Sd = 2 * a.typ_nlocc[S.e_t[e]] + 1, sp2 = plane_stride(Sd);
    const int4 b = a.rep_box[r];
    const int ox = S.gi - (int)(short)(b.x & 0xffff), oy = S.gj - (int)(short)(b.y & 0xffff),
              oz = S.gk - (int)(short)(b.z & 0xffff);  // window -> ball coordinates
    const double *U = a.dtab + a.rep_off[r];
    const double *uk = uf + (size_t)S.e_k[e] * PM * NW;
    double ax = 0.0, ay = 0.0, az = 0.0;
#pragma unroll 4
    for (int i = lane; i < vol; i += 32) {
      const int yz = i / bx, x = x0 + i - yz * bx, zz = yz / by, y = y0 + yz - zz * by, z = z0 + zz;
      const int w = z * VP + y * NP + x + sh;
      for (int q = 0; q < np; q++) {
        const double u = uk[SQB_IDX((size_t)q * NW + w, (size_t)PM * NW, a.status)];
        const long long o = (long long)(q * Sd + oz + z) * sp2 + (oy + y) * Sd + ox + x;
        const double *d = U + SQB_IDX(o, a.dtab_stride - a.rep_off[r], a.status);
        ax += u * d[0];
        ay += u * d[a.dtab_stride];
        az += u * d[2 * a.dtab_stride];
      }
    }
    ax = warp_sum(ax);
    ay = warp_sum(ay);
    az = warp_sum(az);
    if (lane == 0) {
      double *ga = a.g_atoms + (size_t)S.e_atom[e] * 3;
      atomicAdd(ga, ax * iz);
      atomicAdd(ga + 1, ay * iz);
      atomicAdd(ga + 2, az * iz);
    }
  }
}

// The adjoint over the listed nodes (bounds from chi, zee; weights dL/dmu from gmu).
template <int PM, int MAXT, int RY, int MINB>
__global__ void __launch_bounds__(MAXT, MINB) sweep_vjp_kernel(SweepArgs a) {
  extern __shared__ __align__(128) unsigned char smem[];
  Shared &S = *reinterpret_cast<Shared *>(smem);
  unsigned char *dyn = smem + shared_fixed();
  double *pcur = reinterpret_cast<double *>(dyn + planes_bytes(a.n, RY) + ring_bytes(MAXT, RY));
  for (int i = threadIdx.x; i < a.n_gproj + PM; i += blockDim.x) pcur[i] = 0.0;  // [n_gproj..]: the empty id
  double *t0 = a.vjp + (size_t)blockIdx.x * a.vjp_stride;
  for (int i = threadIdx.x; i < (int)vec_points(a.n); i += blockDim.x) t0[i] = 0.0;
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
    node_vjp<PM, RY, MAXT>(a, S, dyn, pcur, a.chi[node], a.zee[node], a.gmu + (size_t)node * (a.npl + 1));
    count_proj_points(a, S, a.npl, 1);
    __syncthreads();
  }
}

template <int PM>
struct VjpKernels {
  template <int MAXT, int MINB>
  static const void *get() {
    return reinterpret_cast<const void *>(&sweep_vjp_kernel<PM, MAXT, TILE_RY, MINB>);
  }
};

const void *vjp_kernel(const SweepArgs &a) {
  return a.pmax == 1   ? pick_tile<VjpKernels<1>>(a.n)
         : a.pmax == 3 ? pick_tile<VjpKernels<3>>(a.n)
                       : nullptr;
}

}  // namespace

size_t sweep_vjp_doubles(int n, int npl) {
  const size_t d = npl * (vec_points(n) + 2 * (size_t)MAXP) + vjp_weights(npl);
  return (d + 31) & ~size_t(31);
}

cudaError_t sweep_vjp_per_sm(const SweepArgs &a, int *per_sm) { return tile_setup(vjp_kernel(a), a, per_sm); }

cudaError_t launch_sweep_vjp(const SweepArgs &a, int grid, cudaStream_t s) {
  const void *kernel = vjp_kernel(a);
  cudaError_t e = tile_setup(kernel, a, nullptr);
  if (e != cudaSuccess) return e;
  SweepArgs args = a;
  void *argv[] = {&args};
  return cudaLaunchKernel(kernel, dim3(grid), dim3(a.nsweep), argv, sweep_smem(a.n, a.pmax, a.n_gproj), s);
}

}  // namespace sqb

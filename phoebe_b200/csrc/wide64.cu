// FP64 pair kernel for cells of up to 16 branches, but for few of them with few R3
// vectors (with per-q1 q2 windows and screening masks): the items and folded vertex of wide.cu, all three
// contractions on the FP64 tensor pipe (mma.sync m8n8k4.f64), one warp per q1
// from T to the rates.
//
// Work item = (one q2, 16 q1), 16 warps.  Per b2:
//   stage 1  T(q1; a, c) = sum_r3 e^{-i q1.R3} Dp(q2)[r3][a][b2][c] as a GEMM with
//            q1 on M (two tiles of 8), the (a, c) in quads of 4 complex columns
//            split over the warps and r3 on K.  Every element of Dp is then a B
//            operand of one warp only, loaded straight from L2 (the item's q2
//            slab is shared by all CTAs) one K step ahead; Re and im of the
//            phases are separate A operands, so Dp is read as it stands.
//   stage 2  X(b1, c) = sum_a e1(a, b1) T(a, c), per warp and q1, 16 x 16 x 16
//   stage 3  V(b1, b3) = sum_c X(b1, c) conj(e3(c, b3)).  X leaves stage 2 as
//            accumulator fragments (row lane / 4, complex column lane % 4), which
//            is the A fragment of stage 3 as it stands: no exchange.
// Two T buffers and one barrier per b2.  Bound by the FP64 pipe: at nb = 15, nr3
// = 67 a vertex has 1.8 MFLOP of stage 1 and 1.0 of stages 2 and 3 with padding.
// Measured on a windowed 24^3 slice of 32 q2 (0.27e6 vertices): 48 ms, 14.6 of 37
// TFLOP/s counted without padding; the shared-memory kernel of builder.cu, DFMA
// with all nb^3 of |V|^2 of 4 q1 in shared memory, took 140 ms.
#include <algorithm>
#include <cstdint>

#include "cplx.cuh"
#include "pair_common.cuh"
#include "phx_internal.h"
#include "warp_rates.cuh"
#include "wide.cuh"

using namespace pairc;

namespace {

constexpr int kQ = 16;             // q1 per item = warps
constexpr int kThreads = 32 * kQ;
constexpr int kSmemMax = 227 * 1024;

struct Layout {
  int T, ev, tab, total;   // byte offsets (phases at 0); ev < 0: e3 read from global memory
  int plane;               // complex per q1 of T
};

int kst(int nr3) { return (nr3 + 3) / 4; }

// 0 total: does not fit
Layout make_layout(int nb, int nr3) {
  Layout L{};
  L.plane = nb * nb + (12 - nb * nb % 8) % 8;   // 4 mod 8: the 8 rows of a T store fall in distinct banks
  const int ph = 2 * kst(nr3) * 512, T = 2 * kQ * L.plane * 16, ev = kQ * nb * nb * 16,
            tab = kQ * warprates::table_bytes(nb) + 256;
  for (int with : {1, 0}) {
    const long long x = (long long)ph + T + (with ? ev : 0) + tab;
    if (x > kSmemMax) continue;
    L.T = ph;
    L.ev = with ? ph + T : -1;
    L.tab = ph + T + (with ? ev : 0);
    L.total = (int)x;
    return L;
  }
  return L;
}

template <bool ADAPTIVE>
__global__ void __launch_bounds__(kThreads, 1) wide64_kernel(wide::Args P, Layout L) {
  extern __shared__ __align__(128) unsigned char smem[];
  const MeshArgs& M = P.m;
  const int nb = M.nb, nbb = nb * nb, nr3 = P.nr3, nks = (nr3 + 3) / 4, nq = M.nq;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int lr = lane >> 2, lc = lane & 3;
  double2* ph = reinterpret_cast<double2*>(smem);   // [2][K step][lane] phases (re, im) of rows lr and 8 + lr
  double2* Tb = reinterpret_cast<double2*>(smem + L.T);   // [2][kQ][plane]
  double2* e3s = reinterpret_cast<double2*>(smem + L.ev) + (size_t)warp * nbb;
  int* ctl = reinterpret_cast<int*>(smem + L.tab + kQ * warprates::table_bytes(nb));   // item, then its q1 [kQ]
  warprates::Vertex<double, 2, 4, ADAPTIVE> v(M, smem + L.tab + (size_t)warp * warprates::table_bytes(nb), lane, 1.0);
  const unsigned total = (unsigned)P.q2_count * P.ntiles;
  const int nquads = (nbb + 3) / 4;

  for (;;) {
    __syncthreads();   // the previous item is done with the phases and the item word
    if (tid == 0) {
      unsigned item;
      for (;;) {
        item = atomicAdd(P.counter, 1u);
        if (item >= total) break;
        const int iq2 = P.q2_first + (int)(item / P.ntiles);
        if (wide::tile_live(P, kQ, item % P.ntiles, iq2, mesh_neg(iq2, M.n0, M.n1, M.n2))) break;
      }
      ctl[0] = item < total ? (int)item : -1;
    }
    __syncthreads();
    const int item = ctl[0];
    if (item < 0) break;
    const int j = item / P.ntiles, tl = item % P.ntiles;
    const int iq2 = P.q2_first + j, iq2m = mesh_neg(iq2, M.n0, M.n1, M.n2);
    // phases e^{-i q1.R3} as A fragments (row lane / 4, K lane % 4); 0 beyond nr3
    for (int e = tid; e < 2 * nks * 32; e += kThreads) {
      const int mt = e / (nks * 32), ks = (e / 32) % nks, ln = e & 31, r = 4 * ks + (ln & 3);
      const int idx = tl * kQ + 8 * mt + (ln >> 2);
      double sn = 0.0, cs = 0.0;
      if (r < nr3) {
        const double* q = M.qcart + 3 * (idx < nq ? P.q1_order[idx] : 0);
        sincos(-(q[0] * P.R3[3 * r] + q[1] * P.R3[3 * r + 1] + q[2] * P.R3[3 * r + 2]), &sn, &cs);
      }
      ph[e] = cmk(cs, sn);
    }
    const int idx = tl * kQ + warp;
    const int q1 = idx < nq ? P.q1_order[idx] : -1;
    int inw = 0;   // bit 0: q2 in the window of q1, bit 1: -q2
    if (q1 >= 0 && !(P.skip && P.skip[(size_t)(iq2 - P.skip_base) * nq + q1])) {
      inw |= (!P.win_energy || P.win_energy[iq2] <= P.win_cut[q1]) ? 1 : 0;
      inw |= (!P.win_energy || P.win_energy[iq2m] <= P.win_cut[q1]) ? 2 : 0;
    }
    v.q1 = max(q1, 0);
    v.iq2 = iq2;
    v.iq2m = iq2m;
    v.iq3 = mesh_add(v.q1, iq2, M.n0, M.n1, M.n2);
    v.inw = inw;
    const double2* e1 = M.U + (size_t)v.q1 * nbb;
    const double2* e3 = M.U + (size_t)v.iq3 * nbb;
    if (inw) {
      if (L.ev >= 0) {
        for (int e = lane; e < nbb; e += 32) e3s[e] = e3[e];
        e3 = e3s;
      }
      v.load();
    }
    __syncthreads();
    const double* D = reinterpret_cast<const double*>(P.Dp + (size_t)j * nr3 * nbb * nb);
    const size_t rstep = (size_t)nbb * nb * 2;   // doubles from one r3 to the next
    for (int b2 = 0; b2 < nb; ++b2) {
      double2* T = Tb + (size_t)(b2 & 1) * kQ * L.plane;
      // stage 1: quads warp, warp + 16, ... of 4 complex (a, c)
      {
        double acc[4][2][4];   // [quad][q1 tile][re A: re, im; im A: re, im]
        size_t off[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int x = min(4 * (warp + kQ * i) + (lane >> 3), nbb - 1);   // B column lane / 4: complex x, re or im
          const int a = x / nb, c = x - a * nb;
          off[i] = 2 * ((size_t)(a * nb + b2) * nb + c) + ((lane >> 2) & 1);
#pragma unroll
          for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int t = 0; t < 4; ++t) acc[i][m][t] = 0.0;
        }
        const int n = (nquads - warp + kQ - 1) / kQ;   // quads of this warp (may be 0)
        double b[4], bn[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) b[i] = i < n ? __ldg(D + (size_t)min(lc, nr3 - 1) * rstep + off[i]) : 0.0;
#pragma unroll 2
        for (int ks = 0; ks < nks; ++ks) {
          const double* Dn = D + (size_t)min(4 * min(ks + 1, nks - 1) + lc, nr3 - 1) * rstep;
#pragma unroll
          for (int i = 0; i < 4; ++i) bn[i] = i < n ? __ldg(Dn + off[i]) : 0.0;
          const double2 a0 = ph[ks * 32 + lane], a1 = ph[(nks + ks) * 32 + lane];
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (i < n) {
              dmma(acc[i][0], a0.x, b[i]);
              dmma(acc[i][0] + 2, a0.y, b[i]);
              dmma(acc[i][1], a1.x, b[i]);
              dmma(acc[i][1] + 2, a1.y, b[i]);
            }
#pragma unroll
          for (int i = 0; i < 4; ++i) b[i] = bn[i];
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int x = 4 * (warp + kQ * i) + lc;
          if (x < nbb)
#pragma unroll
            for (int m = 0; m < 2; ++m)
              T[(size_t)(8 * m + lr) * L.plane + x] = cmk(acc[i][m][0] - acc[i][m][3], acc[i][m][1] + acc[i][m][2]);
        }
      }
      // e1 fragments (row b1 = 8 m + lr, K a = 4 ks + lc), ahead of the barrier
      double2 f1[2][4];
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {
          const int a = 4 * ks + lc, b1 = 8 * m + lr;
          f1[m][ks] = inw && a < nb && b1 < nb ? e1[a * nb + b1] : cmk(0.0, 0.0);
        }
      if (inw) v.width_table(v.f2[b2]);
      __syncthreads();
      if (inw) {
        const double* Tq = reinterpret_cast<const double*>(T + (size_t)warp * L.plane);
        double xr[2][4], xi[2][4];
        {
          double acc[2][4][4];
#pragma unroll
          for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int g = 0; g < 4; ++g)
#pragma unroll
              for (int t = 0; t < 4; ++t) acc[m][g][t] = 0.0;
#pragma unroll
          for (int ks = 0; ks < 4; ++ks) {
            const int a = 4 * ks + lc;
            double b[4];
#pragma unroll
            for (int g = 0; g < 4; ++g) {
              const int c = 4 * g + (lane >> 3);
              b[g] = a < nb && c < nb ? Tq[2 * (a * nb + c) + ((lane >> 2) & 1)] : 0.0;
            }
#pragma unroll
            for (int g = 0; g < 4; ++g)
#pragma unroll
              for (int m = 0; m < 2; ++m) {
                dmma(acc[m][g], f1[m][ks].x, b[g]);
                dmma(acc[m][g] + 2, f1[m][ks].y, b[g]);
              }
          }
#pragma unroll
          for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int g = 0; g < 4; ++g) {
              xr[m][g] = acc[m][g][0] - acc[m][g][3];
              xi[m][g] = acc[m][g][1] + acc[m][g][2];
            }
        }
        double acc[2][4][4];
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
          for (int g = 0; g < 4; ++g)
#pragma unroll
            for (int t = 0; t < 4; ++t) acc[m][g][t] = 0.0;
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {
          const int c = 4 * ks + lc;
          double b[4];
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            const int b3 = 4 * g + (lane >> 3);
            b[g] = c < nb && b3 < nb ? reinterpret_cast<const double*>(e3)[2 * (c * nb + b3) + ((lane >> 2) & 1)] : 0.0;
          }
#pragma unroll
          for (int g = 0; g < 4; ++g)
#pragma unroll
            for (int m = 0; m < 2; ++m) {
              dmma(acc[m][g], xr[m][ks], b[g]);
              dmma(acc[m][g] + 2, xi[m][ks], b[g]);
            }
        }
        // V = X conj(e3), |V|^2 over this q1's plane of T
        __syncwarp();
        double* W = reinterpret_cast<double*>(T + (size_t)warp * L.plane);   // [b1][nb]
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            const int b1 = 8 * m + lr, b3 = 4 * g + lc;
            const double re = acc[m][g][0] + acc[m][g][3], im = acc[m][g][2] - acc[m][g][1];
            if (b1 < nb && b3 < nb) W[b1 * nb + b3] = re * re + im * im;
          }
        __syncwarp();
        v.symmetrize(W, nb);
        v.rates(b2, W, nb);
      }
    }
    if (inw) v.flush(P.lw);
  }
}

}  // namespace

namespace wide {

int q1_fp64_mma(int nb, int nr3) { return nb <= 16 && make_layout(nb, nr3).total ? kQ : 0; }

cudaError_t set_attributes_fp64_mma(int nb, int nr3, int smearing) {
  const int bytes = make_layout(nb, nr3).total;
  return smearing == PHX_SMEAR_ADAPTIVE
             ? cudaFuncSetAttribute(wide64_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes)
             : cudaFuncSetAttribute(wide64_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}

cudaError_t launch_fp64_mma(const Args& A, int grid, cudaStream_t st) {
  const Layout L = make_layout(A.m.nb, A.nr3);
  if (!L.total) return cudaErrorInvalidValue;
  if (A.m.smearing == PHX_SMEAR_ADAPTIVE) wide64_kernel<true><<<grid, kThreads, L.total, st>>>(A, L);
  else wide64_kernel<false><<<grid, kThreads, L.total, st>>>(A, L);
  return cudaGetLastError();
}

}  // namespace wide

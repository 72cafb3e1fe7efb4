// What a warp that owns one (q1, q2) vertex does around its contractions in
// the many-branch kernels (wide_split.cu, wide64.cu): tables of q1 and q3,
// symmetrisation of a b2 plane of |V|^2 and its rates
// (src/bte/scattering.cpp:1209-1318, src/bte/ph_scattering.cpp:338-380,466-518).
//
// Lanes form an 8 x 4 grid; lane (lr, lc) owns the cells b1 = lr + 8 i (i < TR),
// b3 = lc + 4 k (k < TC) of a plane W[b1][ldw].  The three processes of a cell
// are one formula, delta(E_A + E_B - E_C) n_A n_B (n_C + 1), with C = 3 for "+"
// and C = 2, 1 for the two "-" ones.  Live cells are marked with FP32 energies
// against widened bounds and evaluated in FP64 with the reference's own cut-off
// (R = float evaluates the adaptive Gaussian itself in FP32: |V|^2 carries 1e-6).
#pragma once
#include <cstdint>
#include <type_traits>

#include "pair_common.cuh"

namespace warprates {

using namespace pairc;

// W averaged over `count` degenerate blocks (first band f, size z) of the index with stride `step`, a lane
// per value of the other index (stride `line`)
template <class R>
__device__ __forceinline__ void average_blocks(R* W, int line, int step, const uint8_t* f, const uint8_t* z, int count,
                                               int nb, int lane) {
  for (int t = 0; t < count; ++t) {
    const int b = f[t], n = z[t];
    for (int u = lane; u < nb; u += 32) {
      R* w = W + u * line + b * step;
      R sum = 0;
      for (int k = 0; k < n; ++k) sum += w[k * step];
      for (int k = 0; k < n; ++k) w[k * step] = sum / (R)n;
    }
  }
}

// shared memory of one warp's tables
__host__ __device__ inline int table_bytes(int nb) { return (nb * (8 * (4 + 3 + 2 + kMaxT) + 4 * 4 + 6) + 15) / 16 * 16; }

template <class R, int TR, int TC, bool ADAPTIVE>
struct Vertex {
  static constexpr unsigned kAll = 0xffffffffu;
  // bits of a lane's live processes: 3 kinds x TR x TC cells
  static constexpr int kCells = TR * TC;
  using Mask = typename std::conditional<3 * kCells <= 32, unsigned, unsigned long long>::type;
  static constexpr int kBits = 8 * sizeof(Mask), kWords = (3 * kCells + kBits - 1) / kBits;

  const MeshArgs& M;
  const int nb, lane, lr, lc;
  double *E1, *E3, *R1, *R3, *V3, *sq, *acc;   // energies, reciprocals, v3, [nb][+-] squared widths x 6, [nb][kMaxT] sums
  float *F1, *F3, *lim;                        // FP32 energies, [nb][+-] bounds on |e|
  uint8_t *f1, *z1, *f3, *z3, *f2, *z2;        // degenerate blocks: lists for q1 and q3, per band for q2
  double rate0, inv_sigma;
  // the current vertex
  int q1, iq2, iq2m, iq3, inw;                 // inw: bit 0 q2 in the window of q1, bit 1 -q2
  int blocks1, blocks3;
  unsigned take;                               // the lane's states 1 (bits 0..) and 3 (bits 16..) that take part
  float tol;

  __device__ __forceinline__ Vertex(const MeshArgs& m, void* tables, int lane_, double scale)
      : M(m), nb(m.nb), lane(lane_), lr(lane_ >> 2), lc(lane_ & 3) {
    E1 = reinterpret_cast<double*>(tables);
    E3 = E1 + nb;
    R1 = E3 + nb;
    R3 = R1 + nb;
    V3 = R3 + nb;
    sq = V3 + 3 * nb;
    acc = sq + 2 * nb;
    F1 = reinterpret_cast<float*>(acc + nb * kMaxT);
    F3 = F1 + nb;
    lim = F3 + nb;
    f1 = reinterpret_cast<uint8_t*>(lim + 2 * nb);
    z1 = f1 + nb;
    f3 = z1 + nb;
    z3 = f3 + nb;
    f2 = z3 + nb;
    z2 = f2 + nb;
    rate0 = 0.5 * phxc::pi * 0.25 * M.norm * scale;
    inv_sigma = ADAPTIVE ? 0.0 : 1.0 / M.sigma;
  }

  // tables of (q1, q2), q1 >= 0; ends with the warp converged
  __device__ __forceinline__ void load() {
    float em = 0.f;
    for (int b = lane; b < nb; b += 32) {
      const double x1 = M.E[(size_t)q1 * nb + b], x3 = M.E[(size_t)iq3 * nb + b];
      E1[b] = x1;
      E3[b] = x3;
      R1[b] = 1.0 / x1;
      R3[b] = 1.0 / x3;
      F1[b] = (float)x1;
      F3[b] = (float)x3;
      em = fmaxf(em, fmaxf(fabsf((float)x1), fabsf((float)x3)));
      em = fmaxf(em, (float)fmax(fabs(M.E[(size_t)iq2 * nb + b]), fabs(M.E[(size_t)iq2m * nb + b])));
    }
    // three FP32 energies and their sum are within 4.2e-7 of the largest energy of the FP64 one
    tol = 1e-6f * __uint_as_float(__reduce_max_sync(kAll, __float_as_uint(em)));
    if (ADAPTIVE)
      for (int e = lane; e < 3 * nb; e += 32) V3[e] = M.vg[(size_t)iq3 * 3 * nb + e];
    for (int e = lane; e < nb * kMaxT; e += 32) acc[e] = 0.0;
    __syncwarp();
    // forward-scan degenerate blocks (scattering.cpp:1223,1257,1291): those of q1 and q3
    // as lists of the blocks of two and more, those of q2 for every band
    int count = 0;
    if (lane < 3) {
      const double* e = lane == 0 ? E1 : lane == 1 ? E3 : M.E + (size_t)iq2 * nb;
      uint8_t *f = f1 + 2 * lane * nb, *z = f + nb;
      for (int b = 0; b < nb;) {
        const double e0 = e[b];
        int end = b + 1;
        while (end < nb && fabs(e0 - e[end]) < phxc::degThreshold) ++end;
        if (lane < 2) {
          if (end - b > 1) {
            f[count] = (uint8_t)b;
            z[count++] = (uint8_t)(end - b);
          }
        } else {
          for (int k = b; k < end; ++k) {
            f[k] = (uint8_t)b;
            z[k] = (uint8_t)(end - b);
          }
        }
        b = end;
      }
    }
    blocks1 = __shfl_sync(kAll, count, 0);
    blocks3 = __shfl_sync(kAll, count, 1);
    __syncwarp();
    take = 0;
    for (int i = 0; i < TR; ++i)
      if (lr + 8 * i < nb && state_ok(E1[lr + 8 * i])) take |= 1u << i;
    for (int k = 0; k < TC; ++k)
      if (lc + 4 * k < nb && !(E3[lc + 4 * k] < phxc::phEnergyCutoff)) take |= 0x10000u << k;
  }

  // squared widths of (q2 m2, q3 b3) and (-q2 m2, q3 b3) and the bounds on |e|
  // (FP32 square root, widened beyond its error: the evaluation tests exactly)
  __device__ __forceinline__ void width_table(int m2) {
    __syncwarp();   // the previous table has been read
    for (int e = lane; e < 2 * nb; e += 32) {
      if (ADAPTIVE) {
        const double *a = M.vg + ((size_t)(e & 1 ? iq2m : iq2) * nb + m2) * 3, *b = V3 + 3 * (e >> 1);
        const double s2 = width_sq(M.qT, a[0] - b[0], a[1] - b[1], a[2] - b[2]);
        sq[e] = s2;
        lim[e] = s2 == 0.0 ? tol
                           : fmaxf(__fsqrt_rn((float)s2) * (float)(2.0 * 0.4082482904638631 * 1.00001),
                                   (float)(2.0 * phxc::adaptiveCutoff * 1.00001)) + tol;
      } else {
        lim[e] = (float)(6.00001 * M.sigma) + tol;
      }
    }
    __syncwarp();
  }

  // symmetrizeCoupling of a plane: the blocks of b3, then of b1
  __device__ __forceinline__ void symmetrize(R* W, int ldw) {
    if (blocks3) {
      average_blocks(W, ldw, 1, f3, z3, blocks3, nb, lane);
      __syncwarp();
    }
    if (blocks1) {
      average_blocks(W, 1, ldw, f1, z1, blocks1, nb, lane);
      __syncwarp();
    }
  }

  // Rates of plane b2, its member-0 width table in place; the degenerate block
  // of b2 enters as its members' average.
  __device__ __forceinline__ void rates(int b2, const R* W, int ldw) {
    const int nT = M.nT, nq = M.nq, n2 = z2[b2];
#pragma unroll 1
    for (int d2 = 0; d2 < n2; ++d2) {
      const int m2 = f2[b2] + d2;
      const double en2 = M.E[(size_t)iq2 * nb + m2], en2m = M.E[(size_t)iq2m * nb + m2];
      const bool okp = (inw & 1) && state_ok(en2), okm = (inw & 2) && state_ok(en2m);
      if (!okp && !okm) continue;
      if (d2 > 0) width_table(m2);
      const float f2p = (float)en2, f2m = (float)en2m;
      // lower end of e: a Gaussian below x = -27.4 is under the smallest FP64 number
      const float low = (float)(27.4 * M.sigma) + tol;
      const double i2p = rate0 / (en2 * (double)n2), i2m = rate0 / (en2m * (double)n2);
      Mask live[kWords];   // bit kCells kind + TC i + k
#pragma unroll
      for (int u = 0; u < kWords; ++u) live[u] = 0;
      auto mark = [&](int bit) { live[bit / kBits] |= (Mask)1 << (bit % kBits); };
      float x1[TR], dif[TR];
#pragma unroll
      for (int i = 0; i < TR; ++i) {
        const float f = F1[lr + 8 * i];
        x1[i] = f + f2p;
        dif[i] = f - f2m;
      }
#pragma unroll
      for (int k = 0; k < TC; ++k) {
        const float x3 = F3[lc + 4 * k];
        const float2 lm = *reinterpret_cast<const float2*>(lim + 2 * (lc + 4 * k));
#pragma unroll
        for (int i = 0; i < TR; ++i) {
          const float a = x1[i] - x3, b = dif[i] + x3, c = x3 - dif[i];
          if (ADAPTIVE ? fabsf(a) <= lm.x : (a <= lm.x && a >= -low)) mark(TC * i + k);
          if (ADAPTIVE ? fabsf(b) <= lm.y : (b <= lm.y && b >= -low)) mark(kCells + TC * i + k);
          if (ADAPTIVE ? fabsf(c) <= lm.y : (c <= lm.y && c >= -low)) mark(2 * kCells + TC * i + k);
        }
      }
      Mask keep[kWords];
#pragma unroll
      for (int u = 0; u < kWords; ++u) keep[u] = 0;
#pragma unroll
      for (int kd = 0; kd < 3; ++kd)
#pragma unroll
        for (int i = 0; i < TR; ++i) {
          const Mask bits = (take >> i & 1) && (kd ? okm : okp) ? (Mask)(take >> 16) : (Mask)0;
          const int at = kd * kCells + TC * i;
          keep[at / kBits] |= bits << (at % kBits);
          if (at % kBits + TC > kBits) keep[at / kBits + 1] |= bits >> (kBits - at % kBits);
        }
#pragma unroll
      for (int u = 0; u < kWords; ++u) live[u] &= keep[u];
#pragma unroll 1
      for (;;) {
        int t = -1;
#pragma unroll
        for (int u = kWords - 1; u >= 0; --u)
          if (live[u]) t = kBits * u + (sizeof(Mask) == 8 ? __ffsll(live[u]) : __ffs((int)live[u])) - 1;
        if (t < 0) break;
#pragma unroll
        for (int u = 0; u < kWords; ++u)
          if (t / kBits == u) live[u] &= live[u] - 1;
        const int kind = t / kCells, cell = t - kCells * kind, i = cell / TC, k = cell - TC * i;
        const int b1 = lr + 8 * i, b3 = lc + 4 * k;
        const double y1 = E1[b1], y2 = kind ? en2m : en2, y3 = E3[b3];
        const double e = kind == 0 ? y1 + y2 - y3 : kind == 1 ? y1 + y3 - y2 : y2 + y3 - y1;
        double d = (double)W[b1 * ldw + b3] * (kind ? i2m : i2p) * (R1[b1] * R3[b3]);
        if (ADAPTIVE) {
          const double s6 = sq[2 * b3 + (kind ? 1 : 0)] * (1.0 / 6.0);
          double inv = rsqrt(s6), sg = s6 * inv;
          if (sg < phxc::adaptiveCutoff) {
            sg = phxc::adaptiveCutoff;
            inv = 1.0 / phxc::adaptiveCutoff;
          }
          const double x = e * inv;
          const double ex = sizeof(R) == 4 ? (double)expf((float)(-x * x)) : exp(-x * x);
          double g = ex * (inv * (1.0 / (phxc::sqrtPi * phxc::erf2)));
          if (fabs(e) > 2.0 * sg) g = 0.0;
          if (s6 == 0.0) g = e == 0.0 ? 1.0 : 0.0;   // equal velocities
          d *= g;
        } else {
          const double x = e * inv_sigma;
          d *= x > 6.0 ? 0.0 : exp(-x * x) * (inv_sigma * (1.0 / phxc::sqrtPi));
        }
        if (d != 0.0)
          for (int c = 0; c < nT; ++c) {
            const double* B = M.bose + (size_t)c * nq * nb;
            const double n1 = B[(size_t)q1 * nb + b1], nn2 = B[(size_t)(kind ? iq2m : iq2) * nb + m2],
                         n3 = B[(size_t)iq3 * nb + b3];
            const double a = kind == 2 ? n3 : n1, b = kind == 1 ? n3 : nn2, z = kind == 0 ? n3 : kind == 1 ? nn2 : n1;
            atomicAdd(&acc[b1 * kMaxT + c], d * a * b * (z + 1.0));
          }
      }
    }
  }

  // the vertex's sums into (nq, nb, nT) linewidths
  __device__ __forceinline__ void flush(double* lw) {
    __syncwarp();
    const int nT = M.nT;
    for (int e = lane; e < nb * nT; e += 32) {
      const int b1 = e / nT, c = e % nT;
      const double v = acc[b1 * kMaxT + c];
      if (v != 0.0) atomicAdd(&lw[((size_t)q1 * nb + b1) * nT + c], v);
    }
  }
};

}  // namespace warprates

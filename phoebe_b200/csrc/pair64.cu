// Plain FP64 pair builder of the 6-branch cells: linewidths and the
// scattering-matrix modes of PhScatteringMatrix::builder
// (src/bte/ph_scattering.cpp:60-613) on a full Gamma-centred mesh.
//
// The algebra is the one stated at the top of builder.cu (folded vertex
// Dp(q2), one "+" vertex per (q1, q2) that also serves the "-" process of
// (q1, -q2)).  Per (q1, q2):
//   T(a,b2,c)   = sum_r3 e^{-i q1.R3} Dp(q2)[r3][a][b2][c]   74 kFLOP (nr3 = 43)
//   X(b1,b2,c)  = sum_a e1(a,b1) T(a,b2,c)                   10 kFLOP
//   V(b1,b2,b3) = sum_c X(b1,b2,c) conj(e3(c,b3))            10 kFLOP
// so the R3 transform bounds the kernel, and it runs on mma.sync m8n8k4.f64:
// the FP64 tensor pipe reaches 36.9 TFLOP/s here against 26 for DFMA
// streams, and one B operand from shared memory feeds two MMAs.
//
// Layout.  A warp owns 8 q1 (the M rows).  Columns are taken 12 complex
// (b2,c) at a time (two b2), in 3 groups of 4; the six a of a group are six
// 8-column MMA tiles (re and im interleaved), so a thread ends up with T of
// one (q1, b2, c) for all a and the e1 contraction needs no exchange.  X
// passes through shared memory once; in the e3 contraction a thread owns
// three rows (b2, b1) of one q1, and keeps |V|^2 of their six b3 in
// registers through symmetrisation, liveness and rates.  Re and im of the
// phases are separate A operands with their own accumulators, combined per
// thread afterwards, so the image of Dp holds every number once.
// Blocks: 8 such warps (64 q1).  The q2 images are streamed with
// cp.async.bulk, one 17 KB group per stage at nr3 = 43; the last warp to
// have read a stage refills it (a ninth warp for that would cost a quarter of
// the registers: they are granted to warps in fours).
//
// Rates.  A thread marks which of its 3 x 18 processes have a non-zero delta
// and evaluates those, in a fixed order into its own sums: no atomics, so a
// linewidth does not vary between runs.  The three processes of a vertex are
// one formula, delta(E_A + E_B - E_C) n_A n_B (n_C + 1), so lanes at different
// ones do not diverge.
//
// Measured at 16^3, adaptive, 3 temperatures (16.8e6 pairs): 108 ms of pair
// kernel, 14.8 of 37 TFLOP/s over the counted FLOPs, where one thread per (q1,
// b2) on DFMA (255 registers, spills, 6 warps per SM) took 500 ms.  Left out one
// after the other in a copy: the R3 transform alone is 41 ms (31 TFLOP/s), the
// two contractions 18 ms, the marking 18 ms, the rates 31 ms.  Rates through a
// warp-wide queue of live processes took 71 ms instead: filling it and reading
// the results back cost more than the lanes it filled (1.1 live processes a
// thread on average, 3.9 in the busiest).
//
// Degenerate blocks of b1 and b3 are averaged in registers; those of b2 enter
// through the rates: with S the block average, sum_b2 (S W) F = sum_b2 W (S F).
// The members' shares of an element (q1 b1, q2 b2) are summed by the warp (in
// local memory, only at a q2 with degenerate bands) before they go to the
// matrix: an element receives one "+" and one "-" addition onto zero, which
// commute, so it does not vary between runs either.
#include <algorithm>
#include <cstdint>

#include "pair64.cuh"
#include "tc.cuh"

using namespace pairc;

namespace pair64 {
namespace {

constexpr int kNb = 6;
constexpr int kNbb = 36;
constexpr int kWarpsMax = 8;
constexpr int kStages = 2;
constexpr int kStepBytes = 1536;       // one K step of one group: 3 x 32 lanes x 2 doubles
constexpr int kStageStepsMax = 12;
constexpr int kEvStride = 37;          // complex per q1 of the staged eigenvectors (conflict-free 16-byte rows)
constexpr int kXStride = 73;           // complex per q1 of X
constexpr int kSigBytes = 1536;        // widths [8 q1][2 b2][6 b3][+-]
constexpr int kXBytes = 8 * kXStride * 16;
static_assert(18 * 32 * 8 + kSigBytes <= kXBytes, "W and the widths take the place of X");
constexpr int kWarpFixed = 2 * 8 * kEvStride * 16 + kXBytes;
constexpr int kBarBytes = 128;
constexpr int kSmemMax = 227 * 1024;

// K steps of a ring stage: a whole group when it has at most 12
__host__ __device__ inline int stage_steps(int nks) {
  const int n = (nks + kStageStepsMax - 1) / kStageStepsMax;
  return (nks + n - 1) / n;
}
__host__ __device__ inline int warp_bytes(int nks) { return nks * 512 + kWarpFixed; }
int warps_for(int nks) {
  const int w = (kSmemMax - kBarBytes - kStages * stage_steps(nks) * kStepBytes) / warp_bytes(nks);
  return std::max(0, std::min(kWarpsMax, w));
}
size_t smem_bytes(int nks, int warps) {
  return kBarBytes + (size_t)kStages * stage_steps(nks) * kStepBytes + (size_t)warps * warp_bytes(nks);
}

__device__ __forceinline__ void cp16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(tc::smem_u32(dst)), "l"(src) : "memory");
}

__device__ __forceinline__ unsigned count_done(unsigned* p) {
  unsigned old;
  asm volatile("atom.acq_rel.cta.shared::cta.add.u32 %0, [%1], 1;" : "=r"(old) : "r"(tc::smem_u32(p)) : "memory");
  return old;
}

// A wait of this warp gave up: its own copies and the fills issued so far have landed when it
// returns.  The last warp to give up has seen the last fill.
__device__ __noinline__ void give_up(uint64_t* full, int* status) {
  asm volatile("cp.async.wait_all;" ::: "memory");
  volatile unsigned* fills = reinterpret_cast<unsigned*>(full + kStages) + kStages;
  for (int s = 0; s < kStages; ++s) tc::ring_drain(full + s, fills[s], 1, status, 2);
}

// Forward-scan degenerate blocks of six energies, 4 bits per band: its block's first band.
constexpr unsigned kNoBlocks = 0x543210u;
__device__ __forceinline__ unsigned block_starts(const double* e) {
  unsigned s = 0;
  int start = 0;
  double es = e[0];
#pragma unroll
  for (int b = 1; b < kNb; ++b) {
    if (!(fabs(es - e[b]) < phxc::degThreshold)) {
      start = b;
      es = e[b];
    }
    s |= (unsigned)start << (4 * b);
  }
  return s;
}
__device__ __forceinline__ int block_of(unsigned s, int b) { return (s >> (4 * b)) & 7; }
__device__ __forceinline__ int block_size(unsigned s, int b) {
  int n = 0;
#pragma unroll
  for (int k = 0; k < kNb; ++k) n += block_of(s, k) == block_of(s, b);
  return n;
}

// A bound on |e| above which delta(e) is zero, for the marking: the exact test
// is the evaluation's.  FP32 square root, widened beyond its error.
__device__ __forceinline__ double width_limit(double s) {
  constexpr float kFloor = (float)(2.0 * phxc::adaptiveCutoff * 1.00001);
  return s == 0.0 ? 0.0 : (double)fmaxf(__fsqrt_rn((float)s) * (float)(2.0 * 0.4082482904638631 * 1.00001), kFloor);
}

template <bool MAT, bool ADAPTIVE>
__global__ void __launch_bounds__(32 * kWarpsMax, 1) pair64_kernel(Args P, int warps) {
  extern __shared__ __align__(128) unsigned char smem[];
  const MeshArgs& M = P.m;
  const int nks = ksteps(P.nr3), kc = stage_steps(nks), nkc = (nks + kc - 1) / kc;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem);
  unsigned* done = reinterpret_cast<unsigned*>(full + kStages);   // warps that have read a stage, then copies issued to it
  unsigned char* ring = smem + kBarBytes;
  const int stage_bytes = kc * kStepBytes;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int jbeg = blockIdx.y * P.q2_per_slot;
  const int jend = min(P.q2_count, jbeg + P.q2_per_slot);
  // stage i of the slot (group i / nkc from the first group of jbeg on, part i % nkc of its K steps)
  const unsigned nstage = (unsigned)max(0, jend - jbeg) * 9 * nkc;
  auto issue = [&](unsigned i) {
    const unsigned s = i % kStages, g = i / nkc, k = i - g * nkc;
    const uint32_t bytes = min(kc, nks - (int)k * kc) * kStepBytes;
    tc::mbar_arrive_expect_tx(full + s, bytes);
    tc::bulk_g2s(ring + s * stage_bytes,
                 reinterpret_cast<const unsigned char*>(P.img) +
                     (((size_t)jbeg * 9 + g) * nks + (size_t)k * kc) * kStepBytes,
                 bytes, full + s);
    ++done[kStages + s];
  };
  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      tc::mbar_init(full + s, 1);
      done[s] = done[kStages + s] = 0;
    }
    tc::fence_mbar_init();
    for (unsigned i = 0; i < min((unsigned)kStages, nstage); ++i) issue(i);
  }
  __syncthreads();

  unsigned char* mine = ring + kStages * stage_bytes + warp * warp_bytes(nks);
  double2* ph = reinterpret_cast<double2*>(mine);                    // [K step][lane] (re, im)
  double2* e1s = reinterpret_cast<double2*>(mine + nks * 512);       // [8][a][b1]
  double2* e3s = e1s + 8 * kEvStride;                                // [8][c][b3]
  unsigned char* xw = reinterpret_cast<unsigned char*>(e3s + 8 * kEvStride);
  double2* X = reinterpret_cast<double2*>(xw);                       // [8][row (b2l, b1)][c]
  double* w18 = reinterpret_cast<double*>(xw);                       // [18][lane] W, after X
  double2* sig = reinterpret_cast<double2*>(xw + kXBytes - kSigBytes);   // [8][2][6] squared widths of + and -

  const int row = lane >> 2, l = lane & 3;     // q1 of the warp; column / quarter of the rows
  const int nq = M.nq, nT = M.nT, n0 = M.n0, n1 = M.n1, n2 = M.n2;
  const int q1base = (blockIdx.x * warps + warp) * 8;
  const bool valid = q1base + row < nq;
  const int q1 = min(q1base + row, nq - 1);
  for (int ks = 0; ks < nks; ++ks) {
    const int r = 4 * ks + l;
    double sn = 0.0, cs = 0.0;
    if (r < P.nr3) {
      const double* q = M.qcart + 3 * q1;
      sincos(-(q[0] * P.R3[3 * r] + q[1] * P.R3[3 * r + 1] + q[2] * P.R3[3 * r + 2]), &sn, &cs);
    }
    ph[ks * 32 + lane] = cmk(cs, sn);
  }
  for (int t = lane; t < 8 * kNbb; t += 32) {
    const int q = t / kNbb, e = t % kNbb;
    e1s[q * kEvStride + e] = M.U[(size_t)min(q1base + q, nq - 1) * kNbb + e];
  }
  // the thread's rows: b2 = 2 pair + (l >> 1), b1 = b1o + {0, 1, 2}
  const int b1o = 3 * (l & 1), b2l = l >> 1;
  double E1[3];
  unsigned s1;
  {
    double e[kNb];
#pragma unroll
    for (int b = 0; b < kNb; ++b) e[b] = M.E[(size_t)q1 * kNb + b];
    s1 = block_starts(e);
#pragma unroll
    for (int i = 0; i < 3; ++i) E1[i] = (l & 1) ? e[3 + i] : e[i];
  }
  const bool any1 = __any_sync(0xffffffffu, s1 != kNoBlocks);
  unsigned ok1 = 0;   // of the 18 (row, b3): rows whose state takes part
#pragma unroll
  for (int i = 0; i < 3; ++i)
    if (valid && state_ok(E1[i])) ok1 |= 0x3fu << (6 * i);
  double acc[3][kMaxT];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int c = 0; c < kMaxT; ++c) acc[i][c] = 0.0;
  const double rate0 = 0.5 * phxc::pi * 0.25 * M.norm, inv_sigma = ADAPTIVE ? 0.0 : 1.0 / M.sigma;
  __syncwarp();

  unsigned it = 0;
  for (int j = jbeg; j < jend; ++j) {
    const int iq2 = P.q2_first + j;
    const int iq2m = mesh_neg(iq2, n0, n1, n2);
    const int iq3 = mesh_add(q1, iq2, n0, n1, n2);
    for (int t = lane; t < 8 * kNbb; t += 32) {
      const int q = t / kNbb, e = t % kNbb;
      const int q3 = __shfl_sync(0xffffffffu, iq3, q * 4);
      cp16(e3s + q * kEvStride + e, M.U + (size_t)q3 * kNbb + e);
    }
    double E3[kNb];
#pragma unroll
    for (int b = 0; b < kNb; ++b) E3[b] = M.E[(size_t)iq3 * kNb + b];
    const unsigned s3 = block_starts(E3);
    const bool any3 = __any_sync(0xffffffffu, s3 != kNoBlocks);
    unsigned s2;
    {
      double e[kNb];
#pragma unroll
      for (int b = 0; b < kNb; ++b) e[b] = M.E[(size_t)iq2 * kNb + b];
      s2 = block_starts(e);
    }
    unsigned ok3 = 0;
#pragma unroll
    for (int b = 0; b < kNb; ++b)
      if (!(E3[b] < phxc::phEnergyCutoff)) ok3 |= 0x1041u << b;
    // (q1 b1o + i, q2 b) of the matrix
    auto add_matrix = [&](int b, int i, int c, double vp, double vm) {
      const size_t rw = (size_t)q1 * kNb + b1o + i;
      double *dp, *dm, sgn;
      if (P.mat_full) {
        dp = P.matP + (size_t)(iq2 * kNb + b) * P.ld + rw;
        dm = P.matP + (size_t)(iq2m * kNb + b) * P.ld + rw;
        sgn = -2.0;
      } else {
        const size_t o = c * P.mat_tstride + (size_t)(j * kNb + b) * P.ld + rw;
        dp = P.matP + o;
        dm = P.matM + o;
        sgn = 2.0;
      }
      // acc takes half of a rate, the matrix all of it
      if (vp != 0.0) atomicAdd(dp, 2.0 * vp);
      if (vm != 0.0) atomicAdd(dm, sgn * vm);
    };
    double msum[MAT ? kNb : 1][2][3][kMaxT];
    if (MAT && s2 != kNoBlocks)
#pragma unroll 1
      for (int b = 0; b < kNb; ++b)
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int c = 0; c < kMaxT; ++c) msum[b][0][i][c] = msum[b][1][i][c] = 0.0;

#pragma unroll 1
    for (int p = 0; p < 3; ++p) {
      // R3 transform and e1 contraction of the 12 (b2,c) columns
#pragma unroll 1
      for (int g = 0; g < 3; ++g) {
        double cr[kNb][2], ci[kNb][2];
#pragma unroll
        for (int a = 0; a < kNb; ++a) cr[a][0] = cr[a][1] = ci[a][0] = ci[a][1] = 0.0;
        for (int k = 0; k < nkc; ++k, ++it) {
          const unsigned s = it % kStages;
          if (!__all_sync(0xffffffffu, tc::mbar_wait(full + s, (it / kStages) & 1, P.status, 2))) {
            give_up(full, P.status);
            return;
          }
          const double2* B = reinterpret_cast<const double2*>(ring + s * stage_bytes) + lane;
          const double2* A = ph + k * kc * 32 + lane;
          const int steps = min(kc, nks - k * kc);
#pragma unroll 2
          for (int ks = 0; ks < steps; ++ks) {
            const double2 f = A[ks * 32];
            const double2 u0 = B[ks * 96], u1 = B[ks * 96 + 32], u2 = B[ks * 96 + 64];
            dmma(cr[0], f.x, u0.x);
            dmma(cr[1], f.x, u0.y);
            dmma(cr[2], f.x, u1.x);
            dmma(cr[3], f.x, u1.y);
            dmma(cr[4], f.x, u2.x);
            dmma(cr[5], f.x, u2.y);
            dmma(ci[0], f.y, u0.x);
            dmma(ci[1], f.y, u0.y);
            dmma(ci[2], f.y, u1.x);
            dmma(ci[3], f.y, u1.y);
            dmma(ci[4], f.y, u2.x);
            dmma(ci[5], f.y, u2.y);
          }
          __syncwarp();
          // the last warp to have read the stage refills it
          if (lane == 0 && count_done(done + s) == (unsigned)warps - 1) {
            done[s] = 0;
            if (it + kStages < nstage) issue(it + kStages);
          }
        }
        // T(a) = (cr.re - ci.im, cr.im + ci.re) of this thread's (b2, c)
        double2 T[kNb];
#pragma unroll
        for (int a = 0; a < kNb; ++a) T[a] = cmk(cr[a][0] - ci[a][1], cr[a][1] + ci[a][0]);
        const int col = 4 * g + l, cb = col / kNb, c = col - cb * kNb;
        double2* xo = X + row * kXStride + cb * kNbb + c;
        const double2* e1 = e1s + row * kEvStride;
#pragma unroll
        for (int b1 = 0; b1 < kNb; ++b1) {
          double2 x = cmk(0.0, 0.0);
#pragma unroll
          for (int a = 0; a < kNb; ++a) cfma(x, e1[a * kNb + b1], T[a]);
          xo[b1 * kNb] = x;
        }
      }
      if (p == 0) asm volatile("cp.async.wait_all;" ::: "memory");
      __syncwarp();
      // |V|^2 of the thread's three rows and all b3
      double W[3][kNb];
      {
        const double2* x = X + row * kXStride + 3 * l * kNb;
        const double2* e3 = e3s + row * kEvStride;
        double2 xr[3][kNb];
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int c = 0; c < kNb; ++c) xr[i][c] = x[i * kNb + c];
#pragma unroll
        for (int b3 = 0; b3 < kNb; ++b3) {
          double2 v[3];
#pragma unroll
          for (int i = 0; i < 3; ++i) v[i] = cmk(0.0, 0.0);
#pragma unroll
          for (int c = 0; c < kNb; ++c) {
            const double2 e = e3[c * kNb + b3];
#pragma unroll
            for (int i = 0; i < 3; ++i) cfmac(v[i], xr[i][c], e);
          }
#pragma unroll
          for (int i = 0; i < 3; ++i) W[i][b3] = v[i].x * v[i].x + v[i].y * v[i].y;
        }
      }
      if (any3) {
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          double t[kNb];
#pragma unroll
          for (int b = 0; b < kNb; ++b) {
            double s = 0.0;
            int n = 0;
#pragma unroll
            for (int k = 0; k < kNb; ++k)
              if (block_of(s3, k) == block_of(s3, b)) {
                s += W[i][k];
                ++n;
              }
            t[b] = s / (double)n;
          }
#pragma unroll
          for (int b = 0; b < kNb; ++b) W[i][b] = t[b];
        }
      }
      if (any1) {
#pragma unroll
        for (int b3 = 0; b3 < kNb; ++b3) {
          double w[kNb];
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            const double o = __shfl_xor_sync(0xffffffffu, W[i][b3], 1);
            w[i] = (l & 1) ? o : W[i][b3];
            w[3 + i] = (l & 1) ? W[i][b3] : o;
          }
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            const int b = b1o + i;
            double s = 0.0;
            int n = 0;
#pragma unroll
            for (int k = 0; k < kNb; ++k)
              if (block_of(s1, k) == block_of(s1, b)) {
                s += w[k];
                ++n;
              }
            W[i][b3] = s / (double)n;
          }
        }
      }
      __syncwarp();   // X is dead: W (a column per thread) and the widths take its place

      // the members of the b2 block (one, unless E2 is degenerate)
      const int b2 = 2 * p + b2l;
      const int m0 = block_of(s2, b2), mn = block_size(s2, b2);
      {
        const double wgt = 1.0 / (double)mn;
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int b = 0; b < kNb; ++b) w18[(i * kNb + b) * 32 + lane] = W[i][b] * wgt;
      }
      const int members = max(block_size(s2, 2 * p), block_size(s2, 2 * p + 1));
#pragma unroll 1
      for (int mi = 0; mi < members; ++mi) {
        __syncwarp();   // the previous member's widths have been read
        const int mb = min(m0 + mi, kNb - 1);
        const bool member = mi < mn;
        const double E2 = M.E[(size_t)iq2 * kNb + mb], E2m = M.E[(size_t)iq2m * kNb + mb];
        // largest |e| of a live "+" and "-" process for each b3; for a
        // Gaussian the range of e (zero below x = -27.4: under the smallest
        // FP64 number)
        double limp[kNb], limm[kNb];
        double lo;
        if (ADAPTIVE) {
          const double* v2 = M.vg + ((size_t)iq2 * kNb + mb) * 3;
          const double* v2m = M.vg + ((size_t)iq2m * kNb + mb) * 3;
#pragma unroll
          for (int t = 0; t < 3; ++t) {
            const double* v3 = M.vg + ((size_t)iq3 * kNb + b1o + t) * 3;
            sig[(row * 2 + b2l) * kNb + b1o + t] =
                make_double2(width_sq(M.qT, v2[0] - v3[0], v2[1] - v3[1], v2[2] - v3[2]),
                             width_sq(M.qT, v2m[0] - v3[0], v2m[1] - v3[1], v2m[2] - v3[2]));
          }
          __syncwarp();
#pragma unroll
          for (int b = 0; b < kNb; ++b) {
            const double2 t = sig[(row * 2 + b2l) * kNb + b];
            limp[b] = width_limit(t.x);
            limm[b] = width_limit(t.y);
          }
          lo = 0.0;
        } else {
#pragma unroll
          for (int b = 0; b < kNb; ++b) limp[b] = limm[b] = 6.000001 * M.sigma;
          lo = -27.4 * M.sigma;
        }
        auto live = [&](double e, double lim) { return ADAPTIVE ? fabs(e) <= lim : e <= lim && e >= lo; };
        // live (row, b3), bit 6 i + b3, of the three processes delta(E_A + E_B
        // - E_C): C = 3 is "+", C = 2 and C = 1 the two "-" ones
        unsigned m3 = 0, m2 = 0, m1 = 0;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          const double sum = E1[i] + E2, dif = E1[i] - E2m;
#pragma unroll
          for (int b = 0; b < kNb; ++b) {
            const unsigned bit = 1u << (6 * i + b);
            if (live(sum - E3[b], limp[b])) m3 |= bit;
            if (live(dif + E3[b], limm[b])) m2 |= bit;
            if (live(E3[b] - dif, limm[b])) m1 |= bit;
          }
        }
        const unsigned ok = member ? ok1 & ok3 : 0u;
        m3 &= state_ok(E2) ? ok : 0u;
        m2 &= state_ok(E2m) ? ok : 0u;
        m1 &= state_ok(E2m) ? ok : 0u;
        // rates of the thread's live processes, bit 18 k + 6 i + b3 (k = 0: "+")
        double sp[3][kMaxT], sm[3][kMaxT];
        if (MAT)
#pragma unroll
          for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int c = 0; c < kMaxT; ++c) sp[i][c] = sm[i][c] = 0.0;
#pragma unroll 1
        for (unsigned long long m = m3 | (unsigned long long)m2 << 18 | (unsigned long long)m1 << 36; m; m &= m - 1) {
          const int t = __ffsll(m) - 1, kind = t / 18, ib = t - 18 * kind, i = ib / kNb, b = ib - kNb * i;
          const size_t i1 = (size_t)q1 * kNb + b1o + i, i2 = (size_t)(kind ? iq2m : iq2) * kNb + mb,
                       i3 = (size_t)iq3 * kNb + b;
          const size_t iA = kind == 2 ? i3 : i1, iB = kind == 1 ? i3 : i2, iC = kind == 0 ? i3 : kind == 1 ? i2 : i1;
          const double eA = M.E[iA], eB = M.E[iB], eC = M.E[iC];
          const double e = eA + eB - eC;
          double d = w18[ib * 32 + lane] * rate0 / (eA * eB * eC);
          if (ADAPTIVE) {
            const double2 s2 = sig[(row * 2 + b2l) * kNb + b];
            const double s6 = (kind ? s2.y : s2.x) * (1.0 / 6.0);
            double inv = rsqrt(s6), sg = s6 * inv;
            if (sg < phxc::adaptiveCutoff) {
              sg = phxc::adaptiveCutoff;
              inv = 1.0 / phxc::adaptiveCutoff;
            }
            const double x = e * inv;
            double dl = exp(-x * x) * (inv * (1.0 / (phxc::sqrtPi * phxc::erf2)));
            if (fabs(e) > 2.0 * sg) dl = 0.0;
            if (s6 == 0.0) dl = 1.0;   // a zero velocity difference is live only at e = 0
            d *= dl;
          } else {
            const double x = e * inv_sigma;
            d *= x > 6.0 ? 0.0 : exp(-x * x) * (inv_sigma * (1.0 / phxc::sqrtPi));
          }
#pragma unroll
          for (int c = 0; c < kMaxT; ++c)
            if (c < nT) {
              const double* B = M.bose + (size_t)c * nq * kNb;
              const double r = d * B[iA] * B[iB] * (B[iC] + 1.0);
#pragma unroll
              for (int k = 0; k < 3; ++k)
                if (i == k) {
                  acc[k][c] += r;
                  if (MAT) {
                    if (kind) sm[k][c] += r;
                    else sp[k][c] += r;
                  }
                }
            }
        }
        if (MAT)
#pragma unroll
          for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int c = 0; c < kMaxT; ++c)
              if (c < nT) {
                if (s2 == kNoBlocks) {
                  add_matrix(mb, i, c, sp[i][c], sm[i][c]);
                } else {
                  msum[mb][0][i][c] += sp[i][c];
                  msum[mb][1][i][c] += sm[i][c];
                }
              }
      }
      __syncwarp();   // X may be written again
    }
    if (MAT && s2 != kNoBlocks)
#pragma unroll 1
      for (int b = 0; b < kNb; ++b)
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int c = 0; c < kMaxT; ++c)
            if (c < nT) {
              // this thread's b2 and the other half's: one lane adds "+", the other "-"
              const double vp = msum[b][0][i][c] + __shfl_xor_sync(0xffffffffu, msum[b][0][i][c], 2);
              const double vm = msum[b][1][i][c] + __shfl_xor_sync(0xffffffffu, msum[b][1][i][c], 2);
              add_matrix(b, i, c, b2l ? 0.0 : vp, b2l ? vm : 0.0);
            }
  }
  // the two b2 halves of a row's sums, then this block's slot
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int c = 0; c < kMaxT; ++c) {
      const double s = acc[i][c] + __shfl_xor_sync(0xffffffffu, acc[i][c], 2);
      if (valid && b2l == 0 && c < nT)
        P.partial[(((size_t)blockIdx.y * nq + q1) * kNb + b1o + i) * nT + c] += s;
    }
}

// Operand image of the folded vertex, for 8 consecutive q2 and one r3 per
// block: the R2 sum of every (a,b,c) for the 8 q2 at once (an FC3 element is
// read once for 8 phases), then the e2 contraction from shared memory, with
// the q2 phases.  r3 >= nr3 (padding of the last K step) writes zeros.
constexpr int kFoldQ = 8;
constexpr int kFoldR2 = 96;   // R2 phases held at a time
constexpr size_t kFoldSmem = sizeof(double2) * (kFoldQ * (kFoldR2 + kNbb + kNb * kNbb) + kFoldQ);
static_assert(kFoldSmem <= 48 * 1024, "no opt-in needed");
__global__ void __launch_bounds__(256) fold64_kernel(int nr2, int nr3, const double* __restrict__ D3w,
                                                     const double* __restrict__ R2, const double* __restrict__ R3,
                                                     const double* __restrict__ qcart, const double2* __restrict__ U,
                                                     int q2_first, int q2_count, double* __restrict__ img) {
  constexpr int nb3 = kNb * kNbb;
  extern __shared__ __align__(16) char sraw[];
  double2* ph2 = reinterpret_cast<double2*>(sraw);   // [kFoldQ][kFoldR2]
  double2* e2 = ph2 + kFoldQ * kFoldR2;              // [kFoldQ][b][b2]
  double2* Y = e2 + kFoldQ * kNbb;                   // [kFoldQ][a][b][c]
  double2* p3 = Y + kFoldQ * nb3;                    // [kFoldQ]
  const int r3 = blockIdx.x, nks = ksteps(nr3);
  const int j0 = blockIdx.y * kFoldQ;
  const int nj = min(kFoldQ, q2_count - j0);
  const bool pad = r3 >= nr3;
  if (!pad) {
    for (int e = threadIdx.x; e < kFoldQ * kNbb; e += blockDim.x) {
      const int jl = e / kNbb;
      e2[e] = jl < nj ? U[(size_t)(q2_first + j0 + jl) * kNbb + e % kNbb] : cmk(0.0, 0.0);
    }
    if (threadIdx.x < kFoldQ && (int)threadIdx.x < nj) {
      const double* q = qcart + 3 * (q2_first + j0 + threadIdx.x);
      double sn3, cs3;
      sincos(-(q[0] * R3[3 * r3] + q[1] * R3[3 * r3 + 1] + q[2] * R3[3 * r3 + 2]), &sn3, &cs3);
      p3[threadIdx.x] = cmk(cs3, sn3);
    }
    const double* d0 = D3w + (size_t)r3 * nr2 * nb3 + min((int)threadIdx.x, nb3 - 1);
    double2 acc[kFoldQ];
#pragma unroll
    for (int jl = 0; jl < kFoldQ; ++jl) acc[jl] = cmk(0.0, 0.0);
    for (int r0 = 0; r0 < nr2; r0 += kFoldR2) {
      const int nr = min(kFoldR2, nr2 - r0);
      __syncthreads();
      for (int e = threadIdx.x; e < kFoldQ * nr; e += blockDim.x) {
        const int jl = e / nr, r = r0 + e % nr;
        double2 v = cmk(0.0, 0.0);
        if (jl < nj) {
          const double* q = qcart + 3 * (q2_first + j0 + jl);
          double sn, cs;
          sincos(q[0] * R2[3 * r] + q[1] * R2[3 * r + 1] + q[2] * R2[3 * r + 2], &sn, &cs);
          v = cmk(cs, sn);
        }
        ph2[jl * kFoldR2 + r - r0] = v;
      }
      __syncthreads();
#pragma unroll 4
      for (int r = 0; r < nr; ++r) {
        const double x = __ldg(d0 + (size_t)(r0 + r) * nb3);
#pragma unroll
        for (int jl = 0; jl < kFoldQ; ++jl) {
          const double2 p = ph2[jl * kFoldR2 + r];
          acc[jl].x = fma(x, p.x, acc[jl].x);
          acc[jl].y = fma(x, p.y, acc[jl].y);
        }
      }
    }
    if (threadIdx.x < nb3)
#pragma unroll
      for (int jl = 0; jl < kFoldQ; ++jl) Y[jl * nb3 + threadIdx.x] = acc[jl];
    __syncthreads();
  }
  const int ks = r3 >> 2, kl = r3 & 3;
  for (int e = threadIdx.x; e < nj * nb3; e += blockDim.x) {
    const int jl = e / nb3, rest = e % nb3;
    const int a = rest / kNbb, i = rest % kNbb, b2 = i / kNb, c = i % kNb;
    double2 d = cmk(0.0, 0.0);
    if (!pad) {
      const double2* y = Y + jl * nb3 + a * kNbb + c;
      const double2* u = e2 + jl * kNbb + b2;
      double2 z = cmk(0.0, 0.0);
#pragma unroll
      for (int b = 0; b < kNb; ++b) cfma(z, u[b * kNb], y[b * kNb]);
      d = cmul(z, p3[jl]);
    }
    double* o = img + ((((size_t)(j0 + jl) * 9 + (i >> 2)) * nks + ks) * 3 + (a >> 1)) * 64 + (a & 1);
    const int lane = (i & 3) * 8 + kl;
    o[2 * lane] = d.x;
    o[2 * (lane + 4)] = d.y;
  }
}

}  // namespace

int tile_q1(int nr3) { return 8 * warps_for(ksteps(nr3)); }

namespace {
using Kernel = void (*)(Args, int);
Kernel kernel_for(bool matrix, bool adaptive) {
  return matrix ? (adaptive ? pair64_kernel<true, true> : pair64_kernel<true, false>)
                : (adaptive ? pair64_kernel<false, true> : pair64_kernel<false, false>);
}
}  // namespace

cudaError_t set_attributes(int nr3, bool matrix, int smearing) {
  const int nks = ksteps(nr3);
  return cudaFuncSetAttribute(kernel_for(matrix, smearing == PHX_SMEAR_ADAPTIVE),
                              cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes(nks, warps_for(nks)));
}

cudaError_t launch_fold(int nr2, int nr3, const double* D3w, const double* R2, const double* R3, const double* qcart,
                        const double2* U, int q2_first, int q2_count, double* img, cudaStream_t st) {
  const dim3 grid(4 * ksteps(nr3), (q2_count + kFoldQ - 1) / kFoldQ);
  fold64_kernel<<<grid, 256, kFoldSmem, st>>>(nr2, nr3, D3w, R2, R3, qcart, U, q2_first, q2_count, img);
  return cudaGetLastError();
}

cudaError_t launch_pair(const Args& a, int slots, bool matrix, cudaStream_t st) {
  const int nks = ksteps(a.nr3), w = warps_for(nks);
  const dim3 grid((a.m.nq + 8 * w - 1) / (8 * w), slots);
  kernel_for(matrix, a.m.smearing == PHX_SMEAR_ADAPTIVE)<<<grid, 32 * w, smem_bytes(nks, w), st>>>(a, w);
  return cudaGetLastError();
}

}  // namespace pair64

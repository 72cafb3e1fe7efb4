// Split-precision pair kernel for cells with many branches (nb <= 36): the
// same items, image and R3 transform on the tensor cores as wide.cu, with an
// epilogue in which every warp owns one q1.
//
// Per (q1, q2) and b2 the epilogue has 16 nb^3 FLOPs of FP32 contractions and
// nb^2 cells x 3 processes of FP64 energy tests, and nothing of it crosses from
// one q1 to another.  wide.cu's kernel spreads all q1 planes of an item over
// all warps and so separates drain, stage 2, stage 3, symmetrisation, widths
// and rates by block barriers: at nb = 15 these waits were most of its time
// (36 000 cycles per b2 and 8 q1 for about 3 000 of FP32 work).  Here a warp
// takes its q1 from T to the rates alone.  What is left to share is the drain:
// TMEM lanes are rows (a, c), so T of one q1 passes through all warps, which
// meet once per b2 (twice where only one T buffer fits).
//
//   X(b1, c)  = sum_a e1(a, b1) T(a, c)              a warp's lanes form an 8 x 4
//   W(b1, b3) = |sum_c X(b1, c) conj(e3(c, b3))|^2   grid, lane (lr, lc) owning
//                                                    b1 = lr + 8 i, c or b3 = lc + 4 k
// so that every load is 8 or 4 consecutive complex numbers broadcast to the
// rest of the warp.  Loads of rows and columns beyond nb are not guarded: they
// read what follows in shared memory (or the padding of the FP32 eigenvector
// table) into sums that nothing uses.  X takes the place of T's plane and W that of X.
//
// Classes: nb <= 16: 16 warps and q1 (2 x 4 outputs a lane; e1 and e3 of the
// item in shared memory); nb <= 24: 8 q1 (3 x 6); nb <= 36: 8 q1 (5 x 9, 90
// FP32 sums a lane: two warps per scheduler, but 180 FMAs per 14 loads).
// e1 and e3 of the larger cells are read through L1, one row ahead.
// Beyond nb = 36, or where nr3 leaves too little shared memory, wide.cu's runs.
//
// Rates: the lanes' cells are marked with FP32 energies against widened bounds
// (1.3 live of 24 processes in the busiest lane at nb = 15, 3.0 of 135 at nb =
// 36) and the marked ones evaluated in FP64 with the reference's own cut-off.
//
// Measured (24^3 windowed slice of 128 q2, nb = 15, nr3 = 67 / 12^3 slice of 32
// q2, nb = 36, nr3 = 33): 248 -> 74 ms / 114 -> 62 ms a call.  By parts, each
// left out of a copy: A stages and MMAs alone 36 / 17 ms (45 / 27 ms with one K
// step per stage: the handshake of producer and MMA thread costs some 450
// cycles), contractions to 60 / 53 ms, rates the rest.  Packed FMAs were slower
// here (the broadcast operands are register moves): 90 against 85 ms and 65.5
// against 64.2.  Marking in FP64 or tabulating 1/width per plane cost 20 and 30
// ms at nb = 15 (chains of dependent FP64 operations on 4 warps a scheduler).
#include <algorithm>
#include <cstdint>
#include <type_traits>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "cplx.cuh"
#include "pair_common.cuh"
#include "phx_consts.h"
#include "tc.cuh"
#include "wide.cuh"

using namespace pairc;

namespace {

using WideArgs = wide::Args;

constexpr int kKC = 16;                          // K per A stage (one MMA K-step)
constexpr int kMaxStages = 4;
constexpr uint32_t kPart = 128 * kKC * 2;        // one of hi / lo
constexpr uint32_t kStage = 2 * kPart;
constexpr int kItems = 4;
constexpr int kSmemMax = 227 * 1024;

struct Layout {
  int B, T, ev, warp, bars, total;   // byte offsets (A at 0)
  int plane, ldx;                    // complex per q1 of T (and X), row stride of X
  int tb, stages, group;             // T buffers, A stages, K steps per stage
  int warp_bytes;
};

__host__ __device__ inline int mtiles(int nb) { return (nb * nb + 127) / 128; }
__host__ __device__ inline uint32_t tmem_cols(int nb, int nq) {
  const uint32_t need = 2u * mtiles(nb) * 2 * nq;
  uint32_t c = 32;
  while (c < need) c <<= 1;
  return c;
}

// per-warp tables: E1, E3, their reciprocals, v3, 1/width of (q2 m2, -q2 m2),
// sums (doubles); E1, E3 and limits of |e| (floats); blocks (bytes)
__host__ __device__ inline int warp_bytes(int nb) { return (nb * (8 * (4 + 3 + 2 + kMaxT) + 4 * 4 + 6) + 15) / 16 * 16; }

// 0 total: does not fit
Layout make_layout(int nb, int Kp, int nq, bool es) {
  Layout L{};
  L.ldx = nb | 1;
  L.plane = nb * L.ldx;
  L.warp_bytes = warp_bytes(nb);
  // A stages hold several K steps (a handshake of producer and MMA thread costs
  // some 450 cycles, the MMAs of one K step 250): the most that leaves two stages
  const int nkc = Kp / kKC;
  for (int n = (nkc + 5) / 6; n <= nkc; ++n) {
    const int group = (nkc + n - 1) / n;
    for (int tb = 2; tb >= 1; --tb) {
      // two items' phases (hi and lo, 2 nq rows), T, e1 and e3, tables, barriers, slack to align the base
      const size_t sB = (size_t)2 * 2 * (2 * nq) * Kp * 2, sT = ((size_t)tb * nq * L.plane * 8 + 15) / 16 * 16;
      const size_t sE = es ? ((size_t)2 * nq * nb * nb * 8 + 15) / 16 * 16 : 0, sW = (size_t)nq * L.warp_bytes;
      const size_t rest = sB + sT + sE + sW + 512 + 128, stage = (size_t)group * kStage;
      if (rest + 2 * stage > (size_t)kSmemMax) continue;
      L.tb = tb;
      L.group = group;
      L.stages = (int)std::min<size_t>(kMaxStages, (kSmemMax - rest) / stage);
      L.B = L.stages * (int)stage;
      L.T = L.B + (int)sB;
      L.ev = L.T + (int)sT;
      L.warp = L.ev + (int)sE;
      L.bars = L.warp + (int)sW;
      L.total = L.bars + 512 + 128;
      return L;
    }
  }
  L.total = 0;
  return L;
}

__device__ __forceinline__ float fp16_scale(const unsigned* dmax) {
  const float m = __uint_as_float(*dmax);
  if (!(m > 0.f)) return 1.f;
  int e;
  frexpf(m, &e);
  return ldexpf(1.f, -e);
}
__device__ __forceinline__ void split16(double v, bool fp16, uint16_t* hi, uint16_t* lo) {
  if (fp16) {
    const __half h = __double2half(v);
    *hi = __half_as_ushort(h);
    *lo = __half_as_ushort(__double2half(v - (double)__half2float(h)));
  } else {
    const __nv_bfloat16 h = __double2bfloat16(v);
    *hi = __bfloat16_as_ushort(h);
    *lo = __bfloat16_as_ushort(__double2bfloat16(v - (double)__bfloat162float(h)));
  }
}

// is any q1 of the tile paired with q2 or -q2
__device__ bool tile_live(const WideArgs& P, int tile, int iq2, int iq2m) {
  if (!P.win_energy && !P.skip) return true;
  for (int i = 0; i < P.nq1; ++i) {
    const int k = tile * P.nq1 + i;
    if (k >= P.m.nq) break;
    const int q1 = P.q1_order[k];
    if (P.skip && P.skip[(size_t)(iq2 - P.skip_base) * P.m.nq + q1]) continue;
    if (!P.win_energy || P.win_energy[iq2] <= P.win_cut[q1] || P.win_energy[iq2m] <= P.win_cut[q1]) return true;
  }
  return false;
}

__device__ __forceinline__ bool state_ok(double e) { return e >= phxc::phExcludeCutoff && e >= phxc::phEnergyCutoff; }

// s = sum_i (qT_i . dv)^2 of the adaptive width sqrt(s / 6); 0 for equal velocities
__device__ __forceinline__ double width_sq(const double* qT, const double* a, const double* b) {
  const double v0 = a[0] - b[0], v1 = a[1] - b[1], v2 = a[2] - b[2];
  double s = 0.0;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const double d = qT[3 * i] * v0 + qT[3 * i + 1] * v1 + qT[3 * i + 2] * v2;
    s += d * d;
  }
  return s;
}

// W averaged over `count` degenerate blocks (first band f, size z) of the index with stride `step`, a lane
// per value of the other index (stride `line`)
__device__ __forceinline__ void average_blocks(float* W, int line, int step, const uint8_t* f, const uint8_t* z,
                                               int count, int nb, int lane) {
  for (int t = 0; t < count; ++t) {
    const int b = f[t], n = z[t];
    for (int u = lane; u < nb; u += 32) {
      float* w = W + u * line + b * step;
      float sum = 0.f;
      for (int k = 0; k < n; ++k) sum += w[k * step];
      for (int k = 0; k < n; ++k) w[k * step] = sum / (float)n;
    }
  }
}

template <int NQ, int TR, int TC, bool ES, bool ADAPTIVE>
__global__ void __launch_bounds__((NQ + 2) * 32, 1) wide_warp_kernel(WideArgs P, Layout L) {
  constexpr int kN = 2 * NQ;
  // bits of a lane's live processes: 3 kinds x TR x TC cells
  constexpr int kCells = TR * TC;
  using Mask = typename std::conditional<3 * kCells <= 32, unsigned, unsigned long long>::type;
  constexpr int kBits = 8 * sizeof(Mask), kWords = (3 * kCells + kBits - 1) / kBits;
  const MeshArgs& M = P.m;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((128 - (tc::smem_u32(smem_raw) & 127)) & 127);
  const int nb = M.nb, nbb = nb * nb, nr3 = P.nr3, Kp = P.Kp, nkc = Kp / kKC, mt_n = P.mtiles;
  uint8_t* As = smem;
  const int stages = L.stages, group = L.group, ngroups = (nkc + group - 1) / group;
  const uint32_t stage_bytes = (uint32_t)group * kStage;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + L.bars);   // [stages] A stage loaded
  uint64_t* empty = full + kMaxStages;     // [stages] A stage consumed
  uint64_t* tfull = empty + kMaxStages;    // [2] TMEM buffer written by the MMAs
  uint64_t* tfree = tfull + 2;             // [2] TMEM buffer drained by every warp
  uint64_t* bready = tfree + 2;            // [2] phases of an item written by every warp
  uint64_t* bfree = bready + 2;            // [2] phases of an item no longer read by the MMAs
  uint64_t* drained = bfree + 2;           // [2] T buffer written by every warp
  uint64_t* consumed = drained + 2;        // [1] T buffer read by every warp (one buffer only)
  uint64_t* ifull = consumed + 1;          // [kItems]
  uint64_t* iempty = ifull + kItems;       // [kItems]
  uint64_t* done = iempty + kItems;
  volatile int* items = reinterpret_cast<volatile int*>(done + 1);
  uint32_t* tslot = reinterpret_cast<uint32_t*>(done + 1) + kItems;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tslot + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const unsigned total = (unsigned)P.q2_count * P.ntiles;
  const uint32_t tcols = tmem_cols(nb, NQ), bufcols = (uint32_t)mt_n * kN;
  const uint32_t bBytes = (uint32_t)kN * Kp * 2;   // one of hi / lo

  if (tid == 0) {
    for (int i = 0; i < stages; ++i) {
      tc::mbar_init(&full[i], 1);
      tc::mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      tc::mbar_init(&tfull[i], 1);
      tc::mbar_init(&tfree[i], NQ);
      tc::mbar_init(&bready[i], NQ);
      tc::mbar_init(&bfree[i], 1);
      tc::mbar_init(&drained[i], NQ);
    }
    tc::mbar_init(consumed, NQ);
    for (int i = 0; i < kItems; ++i) {
      tc::mbar_init(&ifull[i], 1);
      tc::mbar_init(&iempty[i], NQ + 1);
    }
    tc::mbar_init(done, 1);
    *abort_flag = 0;
    tc::fence_mbar_init();
  }
  if (warp == 0) {
    tc::tmem_alloc(tslot, tcols);
    tc::tmem_relinquish();
  }
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem = *tslot;

  if (warp == NQ) {
    // ---------------- producer: work queue and A tiles ----------------
    if (lane == 0) {
      int st = 0;
      uint32_t par = 1;   // parity of the next wait for an empty stage
      for (int n = 0;; ++n) {
        const int slot = n % kItems;
        if (!tc::mbar_wait_sleep(&iempty[slot], ((n / kItems) & 1) ^ 1, P.status, 1 << 8)) {
          *abort_flag = 1;
          break;
        }
        unsigned item;
        for (;;) {
          item = *abort_flag ? total : atomicAdd(P.counter, 1u);
          if (item >= total) break;
          const int iq2 = P.q2_first + (int)(item / P.ntiles);
          if (tile_live(P, item % P.ntiles, iq2, mesh_neg(iq2, M.n0, M.n1, M.n2))) break;
        }
        items[slot] = item < total ? (int)item : -1;
        tc::mbar_arrive(&ifull[slot]);
        if (item >= total) break;
        const uint8_t* src = P.img + (size_t)(item / P.ntiles) * nb * mt_n * nkc * kStage;
        bool ok = true;
        for (int i = 0; i < nb * mt_n && ok; ++i)
          for (int g = 0; g < ngroups; ++g) {
            if (!tc::mbar_wait(&empty[st], par, P.status, 1 << 9)) {
              ok = false;
              break;
            }
            const uint32_t bytes = min(group, nkc - g * group) * kStage;
            tc::mbar_arrive_expect_tx(&full[st], bytes);
            tc::bulk_g2s(As + st * stage_bytes, src, bytes, &full[st]);
            src += bytes;
            if (++st == stages) {
              st = 0;
              par ^= 1;
            }
          }
        if (!ok) {
          *abort_flag = 1;
          break;
        }
      }
    }
  } else if (warp == NQ + 1) {
    // ---------------- MMA issuer ----------------
    if (lane == 0) {
      const uint32_t idesc = P.fp16 ? tc::idesc_f16_f32(128, kN) : tc::idesc_bf16_f32(128, kN);
      const uint32_t sbB = (uint32_t)(Kp / 8) * 128;
      int st = 0, s = 0;
      uint32_t par = 0;   // parity of the next wait for a full stage
      bool ok = true;
      for (int n = 0; ok; ++n) {
        const int slot = n % kItems;
        if (!tc::mbar_wait_sleep(&ifull[slot], (n / kItems) & 1, P.status, 1 << 10)) { ok = false; break; }
        const int item = items[slot];
        tc::mbar_arrive(&iempty[slot]);
        if (item < 0) break;
        const int bb = n & 1;
        if (!tc::mbar_wait_sleep(&bready[bb], (n >> 1) & 1, P.status, 1 << 11)) { ok = false; break; }
        tc::tc_fence_after();
        const uint32_t bHi = tc::smem_u32(smem + L.B + (size_t)bb * 2 * bBytes), bLo = bHi + bBytes;
        for (int b2 = 0; b2 < nb && ok; ++b2, ++s) {
          const int buf = s & 1;
          if (!tc::mbar_wait_sleep(&tfree[buf], ((s >> 1) & 1) ^ 1, P.status, 1 << 12)) { ok = false; break; }
          tc::tc_fence_after();
          for (int mt = 0; mt < mt_n && ok; ++mt) {
            const uint32_t d = tmem + (uint32_t)buf * bufcols + (uint32_t)mt * kN;
            for (int g = 0; g < ngroups; ++g) {
              if (!tc::mbar_wait(&full[st], par, P.status, 1 << 13)) {
                ok = false;
                break;
              }
              tc::tc_fence_after();
              const int steps = min(group, nkc - g * group);
              for (int k = 0; k < steps; ++k) {
                const int kc = g * group + k;
                const uint32_t aHi = tc::smem_u32(As + st * stage_bytes + k * kStage), aLo = aHi + kPart;
                const uint64_t dAh = tc::smem_desc(aHi, 128, 256), dAl = tc::smem_desc(aLo, 128, 256);
                const uint64_t dBh = tc::smem_desc(bHi + kc * 256, 128, sbB);
                const uint64_t dBl = tc::smem_desc(bLo + kc * 256, 128, sbB);
                tc::mma_bf16(d, dAh, dBh, idesc, kc != 0);
                tc::mma_bf16(d, dAh, dBl, idesc, 1);
                tc::mma_bf16(d, dAl, dBh, idesc, 1);
              }
              tc::mma_commit(&empty[st]);
              if (++st == stages) {
                st = 0;
                par ^= 1;
              }
            }
          }
          if (ok) tc::mma_commit(&tfull[buf]);
        }
        if (ok) tc::mma_commit(&bfree[bb]);
      }
      if (!ok) *abort_flag = 1;
      tc::mma_commit(done);
      tc::mbar_wait_sleep(done, 0, P.status, 1 << 14);
    }
  } else {
    // ---------------- epilogue: warp w owns q1 number w of the item ----------------
    const unsigned kAll = 0xffffffffu;
    const int qd = warp & 3, grp = warp >> 2;
    const int lr = lane >> 2, lc = lane & 3;
    const int nT = M.nT, nq = M.nq;
    constexpr bool adaptive = ADAPTIVE;
    const double sc = P.fp16 ? (double)fp16_scale(P.dmax) : 1.0;
    const double rate0 = 0.5 * phxc::pi * 0.25 * M.norm / (sc * sc);
    const double inv_sigma = adaptive ? 0.0 : 1.0 / M.sigma;
    double* E1 = reinterpret_cast<double*>(smem + L.warp + (size_t)warp * L.warp_bytes);
    double* E3 = E1 + nb;
    double* R1 = E3 + nb;                 // 1 / E1
    double* R3i = R1 + nb;                // 1 / E3
    double* V3 = R3i + nb;
    double* sq = V3 + 3 * nb;             // [nb][+, -] squared widths x 6
    double* acc = sq + 2 * nb;          // [nb][kMaxT]
    float* F1 = reinterpret_cast<float*>(acc + nb * kMaxT);   // E1, E3 in FP32
    float* F3 = F1 + nb;
    float* lim = F3 + nb;                 // [nb][+, -] bounds on |e|
    uint8_t* blk = reinterpret_cast<uint8_t*>(lim + 2 * nb);   // first band and size: q1, q3, q2
    uint8_t *f1 = blk, *z1 = blk + nb, *f3 = blk + 2 * nb, *z3 = blk + 3 * nb, *f2 = blk + 4 * nb, *z2 = blk + 5 * nb;
    float2* e1s = reinterpret_cast<float2*>(smem + L.ev) + (size_t)warp * 2 * nbb;
    float2* e3s = e1s + nbb;
    auto wait = [&](uint64_t* bar, uint32_t parity, int code) -> bool {
      const bool ok = tc::mbar_wait(bar, parity, P.status, code);
      return __all_sync(kAll, ok && !*abort_flag);
    };
    int s = 0;
    for (int n = 0;; ++n) {
      const int slot = n % kItems;
      if (!wait(&ifull[slot], (n / kItems) & 1, 1 << 15)) { *abort_flag = 1; break; }
      const int item = items[slot];
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&iempty[slot]);
      if (item < 0) break;
      const int j = item / P.ntiles, tl = item % P.ntiles;
      const int iq2 = P.q2_first + j, iq2m = mesh_neg(iq2, M.n0, M.n1, M.n2);
      const int idx = tl * NQ + warp;
      const int q1 = idx < nq ? P.q1_order[idx] : -1, q1c = max(q1, 0);
      int inw = 0;   // bit 0: q2 in the window of q1, bit 1: -q2
      if (q1 >= 0 && !(P.skip && P.skip[(size_t)(iq2 - P.skip_base) * nq + q1])) {
        inw |= (!P.win_energy || P.win_energy[iq2] <= P.win_cut[q1]) ? 1 : 0;
        inw |= (!P.win_energy || P.win_energy[iq2m] <= P.win_cut[q1]) ? 2 : 0;
      }
      const int iq3 = mesh_add(q1c, iq2, M.n0, M.n1, M.n2);
      // phases of this q1 into B buffer n & 1, once the MMAs of item n - 2 are done with it
      const int bb = n & 1;
      if (!wait(&bfree[bb], ((n >> 1) & 1) ^ 1, 1 << 16)) { *abort_flag = 1; break; }
      uint8_t* Bh = smem + L.B + (size_t)bb * 2 * bBytes;
      for (int k = lane; k < Kp; k += 32) {
        double re = 0.0, im = 0.0;
        if (k < 2 * nr3) {
          const int r = k < nr3 ? k : k - nr3;
          const double* qc = M.qcart + 3 * q1c;
          double sn, cs;
          sincos(-(qc[0] * P.R3[3 * r] + qc[1] * P.R3[3 * r + 1] + qc[2] * P.R3[3 * r + 2]), &sn, &cs);
          re = k < nr3 ? cs : -sn;   // column 2q: Tr = sum Dr cos - Di sin
          im = k < nr3 ? sn : cs;    // column 2q + 1: Ti = sum Dr sin + Di cos
        }
        uint16_t h, l;
        split16(re, P.fp16 != 0, &h, &l);
        uint32_t off = tc::core_offset(2 * warp, k, Kp, 2);
        *reinterpret_cast<uint16_t*>(Bh + off) = h;
        *reinterpret_cast<uint16_t*>(Bh + bBytes + off) = l;
        split16(im, P.fp16 != 0, &h, &l);
        off = tc::core_offset(2 * warp + 1, k, Kp, 2);
        *reinterpret_cast<uint16_t*>(Bh + off) = h;
        *reinterpret_cast<uint16_t*>(Bh + bBytes + off) = l;
      }
      tc::fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&bready[bb]);
      // tables of this q1 and its q3
      const float2* e1 = ES ? e1s : P.U32 + (size_t)q1c * nbb;
      const float2* e3 = ES ? e3s : P.U32 + (size_t)iq3 * nbb;
      int blocks1 = 0, blocks3 = 0;
      float tol = 0.f;
      unsigned take = 0;   // a lane's states 1 (bits 0..) and 3 (bits 16..) that take part
      if (inw) {
        float em = 0.f;
        for (int b = lane; b < nb; b += 32) {
          const double x1 = M.E[(size_t)q1 * nb + b], x3 = M.E[(size_t)iq3 * nb + b];
          E1[b] = x1;
          E3[b] = x3;
          R1[b] = 1.0 / x1;
          R3i[b] = 1.0 / x3;
          F1[b] = (float)x1;
          F3[b] = (float)x3;
          em = fmaxf(em, fmaxf(fabsf((float)x1), fabsf((float)x3)));
          em = fmaxf(em, (float)fmax(fabs(M.E[(size_t)iq2 * nb + b]), fabs(M.E[(size_t)iq2m * nb + b])));
        }
        // three FP32 energies and their sum are within 4.2e-7 of the largest energy of the FP64 one
        tol = 1e-6f * __uint_as_float(__reduce_max_sync(kAll, __float_as_uint(em)));
        if (adaptive)
          for (int e = lane; e < 3 * nb; e += 32) V3[e] = M.vg[(size_t)iq3 * 3 * nb + e];
        for (int e = lane; e < nb * kMaxT; e += 32) acc[e] = 0.0;
        if (ES)
          for (int e = lane; e < nbb; e += 32) {
            e1s[e] = P.U32[(size_t)q1 * nbb + e];
            e3s[e] = P.U32[(size_t)iq3 * nbb + e];
          }
        __syncwarp();
        // forward-scan degenerate blocks (scattering.cpp:1223,1257,1291): those of q1 and q3
        // as lists of the blocks of two and more, those of q2 for every band
        int count = 0;
        if (lane < 3) {
          const double* e = lane == 0 ? E1 : lane == 1 ? E3 : M.E + (size_t)iq2 * nb;
          uint8_t *f = blk + 2 * lane * nb, *z = f + nb;
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
        for (int i = 0; i < TR; ++i)
          if (lr + 8 * i < nb && state_ok(E1[lr + 8 * i])) take |= 1u << i;
        for (int k = 0; k < TC; ++k)
          if (lc + 4 * k < nb && !(E3[lc + 4 * k] < phxc::phEnergyCutoff)) take |= 0x10000u << k;
      }
      // squared widths of (q2 m2, q3 b3) and (-q2 m2, q3 b3) and the bounds on |e|
      // (FP32 square root, widened beyond its error: the evaluation tests exactly)
      auto width_table = [&](int m2) {
        __syncwarp();   // the previous table has been read
        for (int e = lane; e < 2 * nb; e += 32) {
          if (adaptive) {
            const double s2 = width_sq(M.qT, M.vg + ((size_t)(e & 1 ? iq2m : iq2) * nb + m2) * 3, V3 + 3 * (e >> 1));
            sq[e] = s2;
            lim[e] = s2 == 0.0 ? tol
                               : fmaxf(__fsqrt_rn((float)s2) * (float)(2.0 * 0.4082482904638631 * 1.00001),
                                       (float)(2.0 * phxc::adaptiveCutoff * 1.00001)) + tol;
          } else {
            lim[e] = (float)(6.00001 * M.sigma) + tol;
          }
        }
        __syncwarp();
      };
      bool ok = true;
      for (int b2 = 0; b2 < nb; ++b2, ++s) {
        if (inw) width_table(f2[b2]);
        const int buf = s & 1, tbuf = L.tb == 2 ? buf : 0;
        float2* Tb = reinterpret_cast<float2*>(smem + L.T) + (size_t)tbuf * NQ * L.plane;
        if (L.tb == 1 && s > 0 && !wait(consumed, (s - 1) & 1, 1 << 17)) { ok = false; break; }
        if (!wait(&tfull[buf], (s >> 1) & 1, 1 << 18)) { ok = false; break; }
        tc::tc_fence_after();
        // drain: TMEM lane = row (a, c) of an M tile, columns 2q, 2q + 1 = re, im
        for (int t = grp; t < mt_n * (NQ / 8); t += NQ / 4) {
          const int mt = t / (NQ / 8), cg = t % (NQ / 8);
          float v[16];
          const uint32_t ta = tmem + ((uint32_t)(qd * 32) << 16) + (uint32_t)buf * bufcols + (uint32_t)(mt * kN + cg * 16);
          tc::tmem_ld8(ta, v);
          tc::tmem_ld8(ta + 8, v + 8);
          tc::tmem_wait_ld<16>(v);
          const int row = mt * 128 + qd * 32 + lane;
          if (row < nbb) {
#pragma unroll
            for (int q = 0; q < 8; ++q) Tb[(size_t)(cg * 8 + q) * L.plane + row] = make_float2(v[2 * q], v[2 * q + 1]);
          }
        }
        tc::tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          tc::mbar_arrive(&tfree[buf]);
          tc::mbar_arrive(&drained[tbuf]);
        }
        if (!wait(&drained[tbuf], L.tb == 2 ? (s >> 1) & 1 : s & 1, 1 << 19)) { ok = false; break; }
        if (inw) {
          float2* Tq = Tb + (size_t)warp * L.plane;
          const int ldx = L.ldx;
          float2 w[TR][TC];
          {
            const float2 *pe = e1 + lr, *pt = Tq + lc;
            float2 ev[TR], en[TR];
#pragma unroll
            for (int i = 0; i < TR; ++i) ev[i] = ES ? pe[8 * i] : __ldg(pe + 8 * i);
#pragma unroll
            for (int i = 0; i < TR; ++i)
#pragma unroll
              for (int k = 0; k < TC; ++k) w[i][k] = make_float2(0.f, 0.f);
#pragma unroll 2
            for (int a = 0; a < nb; ++a) {
              if (a + 1 < nb) pe += nb;
#pragma unroll
              for (int i = 0; i < TR; ++i) en[i] = ES ? pe[8 * i] : __ldg(pe + 8 * i);
#pragma unroll
              for (int k = 0; k < TC; ++k) {
                const float2 t = pt[4 * k];
#pragma unroll
                for (int i = 0; i < TR; ++i) cfmaf(w[i][k], ev[i], t);
              }
              pt += nb;
#pragma unroll
              for (int i = 0; i < TR; ++i) ev[i] = en[i];
            }
          }
          __syncwarp();
#pragma unroll
          for (int i = 0; i < TR; ++i)
#pragma unroll
            for (int k = 0; k < TC; ++k)
              if (lr + 8 * i < nb && lc + 4 * k < nb) Tq[(lr + 8 * i) * ldx + lc + 4 * k] = w[i][k];
          __syncwarp();
          {
            const float2 *pe = e3 + lc, *px = Tq + lr * ldx;
            float2 ev[TC], en[TC];
#pragma unroll
            for (int k = 0; k < TC; ++k) ev[k] = ES ? pe[4 * k] : __ldg(pe + 4 * k);
#pragma unroll
            for (int i = 0; i < TR; ++i)
#pragma unroll
              for (int k = 0; k < TC; ++k) w[i][k] = make_float2(0.f, 0.f);
#pragma unroll 2
            for (int c = 0; c < nb; ++c) {
              if (c + 1 < nb) pe += nb;
#pragma unroll
              for (int k = 0; k < TC; ++k) en[k] = ES ? pe[4 * k] : __ldg(pe + 4 * k);
#pragma unroll
              for (int i = 0; i < TR; ++i) {
                const float2 x = px[8 * i * ldx + c];
#pragma unroll
                for (int k = 0; k < TC; ++k) cfmacf(w[i][k], x, ev[k]);
              }
#pragma unroll
              for (int k = 0; k < TC; ++k) ev[k] = en[k];
            }
          }
          __syncwarp();
          float* W = reinterpret_cast<float*>(Tq);   // [b1][ldx]
#pragma unroll
          for (int i = 0; i < TR; ++i)
#pragma unroll
            for (int k = 0; k < TC; ++k)
              if (lr + 8 * i < nb && lc + 4 * k < nb)
                W[(lr + 8 * i) * ldx + lc + 4 * k] = w[i][k].x * w[i][k].x + w[i][k].y * w[i][k].y;
          __syncwarp();
          // symmetrizeCoupling (scattering.cpp:1209-1318): the blocks of b3, then of b1
          if (blocks3) {
            average_blocks(W, ldx, 1, f3, z3, blocks3, nb, lane);
            __syncwarp();
          }
          if (blocks1) {
            average_blocks(W, 1, ldx, f1, z1, blocks1, nb, lane);
            __syncwarp();
          }

          // rates; the block of b2 enters as its members' average
          const int n2 = z2[b2];
#pragma unroll 1
          for (int d2 = 0; d2 < n2; ++d2) {
            const int m2 = f2[b2] + d2;
            const double en2 = M.E[(size_t)iq2 * nb + m2], en2m = M.E[(size_t)iq2m * nb + m2];
            const bool okp = (inw & 1) && state_ok(en2), okm = (inw & 2) && state_ok(en2m);
            if (!okp && !okm) continue;
            if (d2 > 0) width_table(m2);   // member 0's was made before the waits
            const float f2p = (float)en2, f2m = (float)en2m;
            // lower end of e: a Gaussian below x = -27.4 is under the smallest FP64 number
            const float low = (float)(27.4 * M.sigma) + tol;
            const double i2p = rate0 / (en2 * (double)n2), i2m = rate0 / (en2m * (double)n2);
            // live cells, bit kCells kind + TC i + k: processes delta(E_A + E_B - E_C) with C = 3 ("+"), 2, 1 ("-")
            Mask live[kWords];
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
              double d = (double)W[b1 * ldx + b3] * (kind ? i2m : i2p) * (R1[b1] * R3i[b3]);
              if (adaptive) {
                const double s6 = sq[2 * b3 + (kind ? 1 : 0)] * (1.0 / 6.0);
                double inv = rsqrt(s6), sg = s6 * inv;
                if (sg < phxc::adaptiveCutoff) {
                  sg = phxc::adaptiveCutoff;
                  inv = 1.0 / phxc::adaptiveCutoff;
                }
                const double x = e * inv;
                // the Gaussian in FP32 (1e-7): |V|^2 carries 1e-6
                double g = (double)expf((float)(-x * x)) * (inv * (1.0 / (phxc::sqrtPi * phxc::erf2)));
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
                  const double a = kind == 2 ? n3 : n1, b = kind == 1 ? n3 : nn2,
                               z = kind == 0 ? n3 : kind == 1 ? nn2 : n1;
                  atomicAdd(&acc[b1 * kMaxT + c], d * a * b * (z + 1.0));
                }
            }
          }
        }
        __syncwarp();
        if (L.tb == 1 && lane == 0) tc::mbar_arrive(consumed);
      }
      if (!ok) { *abort_flag = 1; break; }
      if (inw)
        for (int e = lane; e < nb * nT; e += 32) {
          const int b1 = e / nT, c = e % nT;
          const double v = acc[b1 * kMaxT + c];
          if (v != 0.0) atomicAdd(&P.lw[((size_t)q1 * nb + b1) * nT + c], v);
        }
      __syncwarp();
    }
  }
  tc::tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc::tc_fence_after();
    tc::tmem_dealloc(tmem, tcols);
  }
}

struct Class {
  int nq, tr, tc;
  bool es;
  void (*fn)(WideArgs, Layout);
};
template <int NQ, int TR, int TC, bool ES>
Class make_class(int smearing) {
  return {NQ, TR, TC, ES,
          smearing == PHX_SMEAR_ADAPTIVE ? wide_warp_kernel<NQ, TR, TC, ES, true> : wide_warp_kernel<NQ, TR, TC, ES, false>};
}
Class class_for(int nb, int smearing) {
  if (nb <= 16) return make_class<16, 2, 4, true>(smearing);
  if (nb <= 24) return make_class<8, 3, 6, false>(smearing);
  return make_class<8, 5, 9, false>(smearing);
}

}  // namespace

namespace wide {

int warp_q1(int nb, int Kp, int* tile_rows) {
  if (nb > 36) return 0;
  const Class c = class_for(nb, PHX_SMEAR_ADAPTIVE);
  if (tile_rows) *tile_rows = c.tr;
  return make_layout(nb, Kp, c.nq, c.es).total ? c.nq : 0;
}

cudaError_t warp_set_attributes(int nb, int Kp, int smearing) {
  const Class c = class_for(nb, smearing);
  const Layout L = make_layout(nb, Kp, c.nq, c.es);
  return cudaFuncSetAttribute(c.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, L.total);
}

cudaError_t launch_warp_split(const Args& A, int grid, cudaStream_t st) {
  const Class c = class_for(A.m.nb, A.m.smearing);
  const Layout L = make_layout(A.m.nb, A.Kp, c.nq, c.es);
  if (!L.total) return cudaErrorInvalidValue;
  c.fn<<<grid, (c.nq + 2) * 32, L.total, st>>>(A, L);
  return cudaGetLastError();
}

}  // namespace wide

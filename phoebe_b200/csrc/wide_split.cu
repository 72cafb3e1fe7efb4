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
// q2, nb = 36, nr3 = 33): 248 -> 75 ms / 114 -> 63 ms a call.  By parts, each
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
#include "half_split.cuh"
#include "pair_common.cuh"
#include "phx_consts.h"
#include "tc.cuh"
#include "warp_rates.cuh"
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

// 0 total: does not fit
Layout make_layout(int nb, int Kp, int nq, bool es) {
  Layout L{};
  L.ldx = nb | 1;
  L.plane = nb * L.ldx;
  L.warp_bytes = warprates::table_bytes(nb);
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

template <int NQ, int TR, int TC, bool ES, bool ADAPTIVE>
__global__ void __launch_bounds__((NQ + 2) * 32, 1) wide_warp_kernel(WideArgs P, Layout L) {
  constexpr int kN = 2 * NQ;
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
      unsigned issued = 0;
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
          if (wide::tile_live(P, P.nq1, item % P.ntiles, iq2, mesh_neg(iq2, M.n0, M.n1, M.n2))) break;
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
            ++issued;
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
      tc::ring_drain(full, issued, stages, P.status, 1 << 9);
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
    const int nq = M.nq;
    const double sc = P.fp16 ? (double)halves::fp16_scale(*P.dmax) : 1.0;
    warprates::Vertex<float, TR, TC, ADAPTIVE> v(M, smem + L.warp + (size_t)warp * L.warp_bytes, lane, 1.0 / (sc * sc));
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
        halves::split16(re, P.fp16 != 0, &h, &l);
        uint32_t off = tc::core_offset(2 * warp, k, Kp, 2);
        *reinterpret_cast<uint16_t*>(Bh + off) = h;
        *reinterpret_cast<uint16_t*>(Bh + bBytes + off) = l;
        halves::split16(im, P.fp16 != 0, &h, &l);
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
      v.q1 = q1c;
      v.iq2 = iq2;
      v.iq2m = iq2m;
      v.iq3 = iq3;
      v.inw = inw;
      if (inw) {
        if (ES)
          for (int e = lane; e < nbb; e += 32) {
            e1s[e] = P.U32[(size_t)q1 * nbb + e];
            e3s[e] = P.U32[(size_t)iq3 * nbb + e];
          }
        v.load();
      }
      bool ok = true;
      for (int b2 = 0; b2 < nb; ++b2, ++s) {
        if (inw) v.width_table(v.f2[b2]);   // ahead of the waits
        const int buf = s & 1, tbuf = L.tb == 2 ? buf : 0;
        float2* Tb = reinterpret_cast<float2*>(smem + L.T) + (size_t)tbuf * NQ * L.plane;
        if (L.tb == 1 && s > 0 && !wait(consumed, (s - 1) & 1, 1 << 17)) { ok = false; break; }
        if (!wait(&tfull[buf], (s >> 1) & 1, 1 << 18)) { ok = false; break; }
        tc::tc_fence_after();
        // drain: TMEM lane = row (a, c) of an M tile, columns 2q, 2q + 1 = re, im
        for (int t = grp; t < mt_n * (NQ / 8); t += NQ / 4) {
          const int mt = t / (NQ / 8), cg = t % (NQ / 8);
          float d[16];
          const uint32_t ta = tmem + ((uint32_t)(qd * 32) << 16) + (uint32_t)buf * bufcols + (uint32_t)(mt * kN + cg * 16);
          tc::tmem_ld8(ta, d);
          tc::tmem_ld8(ta + 8, d + 8);
          tc::tmem_wait_ld<16>(d);
          const int row = mt * 128 + qd * 32 + lane;
          if (row < nbb) {
#pragma unroll
            for (int q = 0; q < 8; ++q) Tb[(size_t)(cg * 8 + q) * L.plane + row] = make_float2(d[2 * q], d[2 * q + 1]);
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
          v.symmetrize(W, ldx);
          v.rates(b2, W, ldx);
        }
        __syncwarp();
        if (L.tb == 1 && lane == 0) tc::mbar_arrive(consumed);
      }
      if (!ok) { *abort_flag = 1; break; }
      if (inw) v.flush(P.lw);
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

// Plain FP64 pair builder of the 6-branch cells (pair64.cu): the fold that
// writes the R3 operand image and the pair kernel on the FP64 tensor pipe.
#pragma once
#include "pair_common.cuh"

namespace pair64 {

// K steps (4 R3 vectors each) of the R3 transform, and the bytes of one q2's
// operand image: [9 column groups][K step][3 pairs of a][32 lanes][2] doubles.
__host__ __device__ inline int ksteps(int nr3) { return (nr3 + 3) / 4; }
inline size_t image_bytes(int nr3) { return (size_t)9 * ksteps(nr3) * 1536; }

struct Args {
  pairc::MeshArgs m;
  int nr3;
  const double* R3;
  const double* img;   // image of the chunk's q2
  int q2_first, q2_count, q2_per_slot;
  double* partial;     // (S, nq, 6, nT): every slot is added to by one block per tile
  // matrix modes: column-major blocks of the scattering matrix, element
  // (row, col) at col * ld + row, row = 6 q1 + b1; added to atomically.
  //   mat_full = 1: matP is the whole matrix (one temperature): the "+" rates
  //     of (q1 b1, q2 b2) and minus the "-" rates of (q1 b1, -q2 b2).
  //   mat_full = 0: zeroed slabs of the chunk, column 6 j + b2 (j = q2 -
  //     q2_first): matP the "+" rates, matM the "-" rates of (q1 b1, -q2 b2),
  //     each temperature mat_tstride elements further on.
  double* matP;
  double* matM;
  long long ld;
  size_t mat_tstride;
  int mat_full;
  int* status;         // a wait that gave up
};

// q1 points per block, 0 when nr3 does not fit in shared memory
int tile_q1(int nr3);
cudaError_t launch_fold(int nr2, int nr3, const double* D3w, const double* R2, const double* R3, const double* qcart,
                        const double2* U, int q2_first, int q2_count, double* img, cudaStream_t st);
cudaError_t launch_pair(const Args& a, int slots, bool matrix, cudaStream_t st);
// shared memory of the pair kernel for this nr3 (before any stream capture)
cudaError_t set_attributes(int nr3, bool matrix, int smearing);
// R3 vectors that the FP64 path takes
constexpr int kMaxR3 = 262;

}  // namespace pair64

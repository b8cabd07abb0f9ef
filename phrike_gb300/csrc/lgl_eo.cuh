// LGL x LGL steps by even and odd parts on the tensor cores (lgl_eo.cu).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

namespace ps {

constexpr int kEoParts = 3;  // bf16 parts of an operand
// N tiles of the contractions; ps_plan_desc.umma_n_tile 64, 128, 176, 256 in turn
constexpr int kEoTiles[4] = {48, 64, 80, 144};

// One axis: n nodes, h = ceil(n/2) mirrored pairs (the centre of an odd n is
// its own mirror), split matrices and the operand pitch.
struct EoAxis {
  int n, h;
  int kp;     // bf16 pitch of operand rows (multiple of 8)
};

// Device buffers of a plan's even/odd steps, P = kEoParts.
struct EoBufs {
  EoAxis x, y;
  void* X;     // x operand  [P][2 (even, odd)][nsolve*4*ny][x.kp]
  void* Y;     // y operand  [P][2][nsolve*4*nx][y.kp]
  float* CX;   // x products [2][nsolve*4*ny][ldx], parity of the operand (the plan's G)
  int ldx;
  float* CY;   // y products [2][nsolve*4][y.h][nx]
  CUtensorMap mX, mY, mDx, mDy, mFx, mFy;
  int ntx;     // N tile of both directions
};

// Split even/odd matrices [P][2][h][kp] of a float64 matrix M [n][n]:
//   even part: M_ij + M_i,n-1-j, odd: M_ij - M_i,n-1-j (an odd n's centre
//   column: 2 M_ic, met by e_c = f_c, and 0)
// (of I - M with complement)
cudaError_t launch_eo_matrix(const double* M, int n, int kp, bool complement, void* out, cudaStream_t s);
int encode_eo_map(CUtensorMap* m, const void* base, int h, int rows, int kp, int box_rows);
// N tile of contractions with h output columns and mt tiles of 128 rows
int eo_n_tile(int h, long mt);

struct EoGemmArgs {
  EoBufs b;
  int nsolve;
  int dirs;            // bit 0: x, bit 1: y
  int filter;          // the filter's complements I - F instead of D
  const int* active;
  int* status;
  int ntiles, stages;  // column tiles, ring depth (set by the launch)
};
cudaError_t launch_eo_gemm(const EoGemmArgs& a, cudaStream_t s);

// Where the state of a launch comes from, and what is made of it.
enum { kEoStart = 0, kEoStage = 1 };
enum { kEoFlux = 0, kEoFilterX = 1, kEoOut = 2 };
struct EoStageArgs {
  EoBufs b;
  const float* U;      // U^n [nsolve][4][ny][nx]
  float* out;          // new state (kEoOut; may be U)
  const float* acc_in; // RK increments so far (stages >= 1)
  float* acc_out;
  float* S;            // filter: the new state [nsolve][4][ny][nx], and
  float* V;            // the state after the x filter
  int nsolve;
  int stage;           // 0..3 of the products in CX, CY
  const double* dt_dev;
  double dt;
  float gamma, rho_min, p_min;
  const float* eref;
  const int* active;
  int rk2;
  int shift_in, shift_out;  // U holds E; out takes E
  int wall_acc;             // keep the wall points' own increments (filter on)
};
// from: kEoStart (U^n itself) or kEoStage; to: kEoFlux, kEoFilterX or kEoOut
cudaError_t launch_eo_stage(const EoStageArgs& a, int from, int to, cudaStream_t s);
// x products of the filter -> y operand; y products -> the state with its walls
cudaError_t launch_eo_filter_y(const EoStageArgs& a, cudaStream_t s);
cudaError_t launch_eo_filter_out(const EoStageArgs& a, cudaStream_t s);

}  // namespace ps

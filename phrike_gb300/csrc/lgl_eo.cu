// LGL x LGL steps by even and odd parts on the tensor cores.
//
// The LGL nodes are symmetric, so the differentiation matrix is
// centro-antisymmetric (D_{n-1-i,n-1-j} = -D_ij) and the nodal filter
// centro-symmetric.  With e_j = f_j + f_{n-1-j} and o_j = f_j - f_{n-1-j},
//   g_i - g_{n-1-i} = sum_{j<h} (D_ij + D_{i,n-1-j}) e_j
//   g_i + g_{n-1-i} = sum_{j<h} (D_ij - D_{i,n-1-j}) o_j
// give D f from two contractions of half the size each way: half the
// multiplications and half the operand traffic of the full product (the
// even-odd decomposition of Solomonoff, J. Comput. Phys. 98, 1992).
//
// Operands are split into three bf16 parts, which hold all 24 bits of a
// float32, and the six products above 2^-24 are taken, accumulating in float32
// in tensor memory.  Both the float32 plans (whose contractions ran on the CUDA
// cores) and the split-bf16 x3 plans step this way; with two parts and three
// products the even and odd sums lose more than the full ones (momentum after
// 500 steps at 513^2 7.9e-5 off against 4.6e-5).  The filter is applied as
// f - (I - F) f, so that only its small complement goes through the product.
//
// An RK stage is two launches, the x and y contractions of all solves,
// components and parities in one, and one cell-wise kernel that turns the
// products into the next stage's operands: stage update, clamp, walls,
// fluxes, even and odd parts, split.  The walls (columns, then rows) give every
// wall point the values of the nearest interior point with the normal
// momentum zero, so they are read through that rule instead of being stored.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "launch.cuh"
#include "lgl_eo.cuh"
#include "pass_common.cuh"
#include "tma.cuh"
#include "umma.cuh"

namespace ps {

namespace {
constexpr int P = kEoParts;

// P-part split: each part the bf16 rounding of what the earlier ones leave
template <typename T>
__device__ __forceinline__ void split_parts(T v, __nv_bfloat16 (&part)[P]) {
#pragma unroll
  for (int p = 0; p < P; ++p) {
    part[p] = __float2bfloat16_rn((float)v);
    v -= (T)__bfloat162float(part[p]);
  }
}
}  // namespace

__global__ void k_eo_matrix(const double* M, int n, int kp, int complement, __nv_bfloat16* out) {
  const int h = (n + 1) / 2;
  const long plane = 2L * h * kp;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < h * h; e += gridDim.x * blockDim.x) {
    const int i = e / h, j = e - i * h, jm = n - 1 - j;
    double a = M[(long)i * n + j], b = M[(long)i * n + jm];
    if (complement) {
      a = (i == j ? 1.0 : 0.0) - a;
      b = (i == jm ? 1.0 : 0.0) - b;
    }
#pragma unroll
    for (int par = 0; par < 2; ++par) {
      __nv_bfloat16 q[P];
      split_parts<double>(par == 0 ? a + b : a - b, q);  // centre column: 2 M_ic (e_c = f_c), 0
#pragma unroll
      for (int p = 0; p < P; ++p) out[p * plane + ((long)par * h + i) * kp + j] = q[p];
    }
  }
}

cudaError_t launch_eo_matrix(const double* M, int n, int kp, bool complement, void* out, cudaStream_t s) {
  k_eo_matrix<<<128, 256, 0, s>>>(M, n, kp, complement ? 1 : 0, static_cast<__nv_bfloat16*>(out));
  return cudaGetLastError();
}

// 4-D map over [P][2][rows][kp] bf16 (innermost first: k < h, rows, parity,
// part), box 64 x box_rows, 128-byte swizzle.
int encode_eo_map(CUtensorMap* m, const void* base, int h, int rows, int kp, int box_rows) {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      f = nullptr;
    return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(f);
  }();
  if (!fn) return -1;
  const cuuint64_t dims[4] = {(cuuint64_t)h, (cuuint64_t)rows, 2, (cuuint64_t)P};
  const cuuint64_t row_b = (cuuint64_t)kp * 2;
  const cuuint64_t strides[3] = {row_b, row_b * rows, row_b * rows * 2};
  const cuuint32_t box[4] = {64, (cuuint32_t)box_rows, 1, 1};
  const cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return (r == CUDA_SUCCESS) ? 0 : (int)r;
}

// N tile for h output columns and mt tiles of 128 rows: waves of CTAs (one per
// SM) times the work of one, its columns plus 128 columns' worth of row operand
// and set-up.  Every output is the same dot product for every tile.  513 nodes
// (257 pairs) alone take 144 columns (136 CTAs, one wave), 257 nodes (129 pairs)
// 48 (108 CTAs).  Of 24 grids and batches from 129 to 1025 nodes, each timed at
// all four, the rule takes the fastest tile; with 64 columns' worth it took 80 for
// 144 at 385^2 x 14 (834 / 748 us per step), 449^2 x 8 (627 / 568) and 769^2 (272 / 210).
int eo_n_tile(int h, long mt) {
  int best = 144;
  long cost = -1;
  for (int nt : kEoTiles) {
    const long waves = (mt * ((h + nt - 1) / nt) + 147) / 148;
    const long c = waves * (nt + 128);
    if (cost < 0 || c < cost) {
      cost = c;
      best = nt;
    }
  }
  return best;
}

// ---------------------------------------------------------------------------
// C[par][m][n] = sum_k A[par][m][k] B[par][n][k]: rows m = (solve, component,
// line) of the operand, n < h.  One CTA per 128 x NT tile, 128 threads:
// thread 0 issues the TMA loads, thread 32 the MMAs, all four warps drain
// TMEM.  blockIdx.x = column tile (fastest) and row tile, since the row tiles
// of a batch pass the 65535 of gridDim.y; blockIdx.z = parity (+ 2 for y).  x
// products are stored as rows of ldx; y products with the lanes along x (rows
// m = (solve, c, i) go to [solve, c][n][i]).
// ---------------------------------------------------------------------------
template <int NT>
struct EoSmem {
  static constexpr int kA = 128 * 128, kB = NT * 128;  // one part: 64 bf16 per row
  static constexpr int kStage = P * (kA + kB);
  static constexpr int ST = (3 * kStage + 1024 <= 226 * 1024) ? 3 : 2;  // ring depth
  static constexpr int bytes(int stages) { return stages * kStage + 1024; }  // + alignment slack
};

template <int NT>
__global__ void __launch_bounds__(128, 1)
    k_eo_gemm(const __grid_constant__ CUtensorMap mAx, const __grid_constant__ CUtensorMap mBx,
              const __grid_constant__ CUtensorMap mAy, const __grid_constant__ CUtensorMap mBy, EoGemmArgs g) {
  using SM = EoSmem<NT>;
  const int ST = g.stages;
  // two accumulators: hi hi products, and the others (2^-8 smaller), so that
  // the leading sum is rounded once per 16 terms and not six times
  constexpr uint32_t COLS = 2 * NT <= 128 ? 128 : 2 * NT <= 256 ? 256 : 512;
  extern __shared__ unsigned char umma_smem_raw[];
  __shared__ uint64_t full[SM::ST], empty[SM::ST], done;
  __shared__ uint32_t tmem_base;
  __shared__ int abort_flag, issued, consumed;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool ydir = (g.dirs == 2) || (g.dirs == 3 && blockIdx.z >= 2);
  const int par = blockIdx.z & 1;
  const EoAxis& ax = ydir ? g.b.y : g.b.x;
  const int line = ydir ? g.b.x.n : g.b.y.n;  // lines per component
  const int M = g.nsolve * 4 * line, N = ax.h;
  const int mt = blockIdx.x / g.ntiles;
  const int m0 = mt * 128, n0 = (blockIdx.x - mt * g.ntiles) * NT;
  if (m0 >= M || n0 >= N) return;
  const CUtensorMap* mA = ydir ? &mAy : &mAx;
  const CUtensorMap* mB = ydir ? &mBy : &mBx;
  const uint32_t raw = smem_addr(umma_smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  unsigned char* sbase = umma_smem_raw + (base - raw);
  if (tid == 0) {
    for (int s = 0; s < ST; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(&done, 1);
    fence_barrier_init();
    abort_flag = 0;
    issued = 0;
    consumed = 0;
  }
  __syncwarp();
  if (warp == 0) {  // whole warp, converged (.sync.aligned)
    tmem_alloc(&tmem_base, COLS);
    tmem_relinquish();
  }
  dep_wait();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_base;
  volatile int* vabort = &abort_flag;
  // a tile whose rows all belong to inactive solves loads and stores nothing
  bool any = g.active == nullptr;
  for (int z = m0 / (4 * line); !any && z <= (min(m0 + 128, M) - 1) / (4 * line); ++z) any = g.active[z] != 0;
  const int nk = any ? (ax.h + 63) / 64 : 0;

  if (tid == 0) {  // producer
    int kb = 0;
    for (; kb < nk; ++kb) {
      const int s = kb % ST;
      if (kb >= ST) {
        const uint32_t ph = ((kb / ST) - 1) & 1;
        bool ok = false;
        for (uint32_t i = 0; i < kMaxPolls && !ok; ++i) {
          ok = mbar_try_wait(&empty[s], ph);
          if (!ok && *vabort) break;
        }
        if (!ok) {
          if (!*vabort) atomicOr(g.status, kStatusTmaTimeout);
          *vabort = 1;
          break;
        }
      }
      if (*vabort) break;
      unsigned char* st = sbase + s * SM::kStage;
      mbar_arrive_expect_tx(&full[s], SM::kStage);
#pragma unroll
      for (int p = 0; p < P; ++p) {
        tma_load_4d(st + p * SM::kA, mA, kb * 64, m0, par, p, &full[s]);
        tma_load_4d(st + P * SM::kA + p * SM::kB, mB, kb * 64, n0, par, p, &full[s]);
      }
    }
    issued = kb;
  } else if (tid == 32) {  // MMA issuer
    constexpr uint32_t idesc = bf16_idesc(128, NT);
    int kb = 0;
    for (; kb < nk; ++kb) {
      const int s = kb % ST;
      const uint32_t ph = (kb / ST) & 1;
      bool ok = false;
      for (uint32_t i = 0; i < kMaxPolls && !ok; ++i) {
        ok = mbar_try_wait(&full[s], ph);
        if (!ok && *vabort) break;
      }
      if (!ok) {
        if (!*vabort) atomicOr(g.status, kStatusTmaTimeout);
        *vabort = 1;
        break;
      }
      tc_fence_after();
      const uint32_t st = base + s * SM::kStage;
      const int rest = ax.h - kb * 64;
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {
        if (kk * 16 >= rest) break;    // what lies past h is zero
        const uint32_t off = kk * 32;  // 16 bf16 along K
        uint64_t dA[P], dB[P];
#pragma unroll
        for (int p = 0; p < P; ++p) {
          dA[p] = sw128_kmajor_desc(st + p * SM::kA + off);
          dB[p] = sw128_kmajor_desc(st + P * SM::kA + p * SM::kB + off);
        }
        // products of parts (a, b) with a + b < P
        const uint32_t first = (kb == 0 && kk == 0) ? 0u : 1u;
        umma_bf16(tmem, dA[0], dB[0], idesc, first);
        umma_bf16(tmem + NT, dA[0], dB[1], idesc, first);
        umma_bf16(tmem + NT, dA[1], dB[0], idesc, 1u);
        umma_bf16(tmem + NT, dA[1], dB[1], idesc, 1u);
        umma_bf16(tmem + NT, dA[0], dB[2], idesc, 1u);
        umma_bf16(tmem + NT, dA[2], dB[0], idesc, 1u);
      }
      umma_commit(&empty[s]);
    }
    consumed = kb;
    umma_commit(&done);
  }
  __syncwarp();
  // epilogue: every thread owns one accumulator row (TMEM lane)
  bool ok = false;
  for (uint32_t i = 0; i < kMaxPolls && !ok; ++i) ok = mbar_try_wait(&done, 0);
  if (!ok) atomicOr(g.status, kStatusTmaTimeout);
  tc_fence_after();
  const int all_ok = __syncthreads_and(ok ? 1 : 0);  // CTA-uniform: TMEM loads are warp-collective
  const bool valid = all_ok && (*vabort == 0) && nk > 0;
  const int m = m0 + warp * 32 + lane;
  if (valid) {
    float* row;    // element n at row[n * step]
    long step;
    if (ydir) {
      const int sc = m / line, i = m - sc * line;
      step = line;
      row = g.b.CY + ((long)(par * g.nsolve * 4 + sc) * N) * line + i;
    } else {
      step = 1;
      row = g.b.CX + ((long)par * M + m) * g.b.ldx;
    }
#pragma unroll 1
    for (int c0 = 0; c0 < NT; c0 += 16) {
      float v[16], w[16];
      tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0, v);
      tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(NT + c0), w);
#pragma unroll
      for (int q = 0; q < 16; ++q) v[q] += w[q];
      if (m >= M) continue;
      if (ydir) {  // lanes along x: whole lines per column
#pragma unroll
        for (int q = 0; q < 16; ++q)
          if (n0 + c0 + q < N) row[(n0 + c0 + q) * step] = v[q];
      } else {     // rows padded to ldx: 16-byte stores (columns past N are zero)
#pragma unroll
        for (int q = 0; q < 16; q += 4)
          if (n0 + c0 + q < g.b.ldx)
            *reinterpret_cast<float4*>(row + n0 + c0 + q) = make_float4(v[q], v[q + 1], v[q + 2], v[q + 3]);
      }
    }
  }
  // drain loads that were issued but never consumed (abort path only)
  if (tid == 0) {
    for (int kb = consumed; kb < issued; ++kb) {
      const int s = kb % ST;
      const uint32_t ph = (kb / ST) & 1;
      for (uint32_t i = 0; i < kMaxPolls; ++i)
        if (mbar_try_wait(&full[s], ph)) break;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem, COLS);
  }
}

namespace {
template <int NT>
cudaError_t eo_gemm_t(EoGemmArgs a, cudaStream_t s) {
  cudaError_t e;
  if ((e = set_smem(k_eo_gemm<NT>, EoSmem<NT>::bytes(EoSmem<NT>::ST))) != cudaSuccess) return e;
  const EoBufs& b = a.b;
  const bool x = a.dirs & 1, y = a.dirs & 2;
  const int rx = x ? a.nsolve * 4 * b.y.n : 0, ry = y ? a.nsolve * 4 * b.x.n : 0;
  const int hx = x ? b.x.h : 0, hy = y ? b.y.h : 0;
  const int rows = rx > ry ? rx : ry, h = hx > hy ? hx : hy;
  a.ntiles = (h + NT - 1) / NT;
  // Up to 64 pairs the dot product is one block and a tile one load, one set of
  // MMAs and one store in turn: with a ring of one stage two or three CTAs share
  // an SM and overlap them (TMEM holds two or three of their accumulators).
  // Steps of float32 batches: 17^2 x 1000 401 -> 292 us, 33^2 x 200 190 -> 138, 65^2 x
  // 64 169 -> 137 (the CUDA-core contractions took 268, 187 and 242).
  a.stages = (h <= 64 && 2 * NT <= 256) ? 1 : EoSmem<NT>::ST;
  const int bytes = EoSmem<NT>::bytes(a.stages);
  const dim3 grid(a.ntiles * ((rows + 127) / 128), 1, (x && y) ? 4 : 2);
  return launch_dep(k_eo_gemm<NT>, grid, 128, bytes, s, b.mX, a.filter ? b.mFx : b.mDx, b.mY,
                    a.filter ? b.mFy : b.mDy, a);
}
}  // namespace

cudaError_t launch_eo_gemm(const EoGemmArgs& a, cudaStream_t s) {
  switch (a.b.ntx) {  // one tile for both directions (maps are encoded with it)
    case kEoTiles[0]: return eo_gemm_t<kEoTiles[0]>(a, s);
    case kEoTiles[1]: return eo_gemm_t<kEoTiles[1]>(a, s);
    case kEoTiles[2]: return eo_gemm_t<kEoTiles[2]>(a, s);
    case kEoTiles[3]: return eo_gemm_t<kEoTiles[3]>(a, s);
    default: return cudaErrorInvalidValue;
  }
}

// ---------------------------------------------------------------------------
// Cell-wise kernel.  A thread holds the four mirror images of one point
// (j, i) of the lower-left quarter; tiles of 32 x 8 such points.
// ---------------------------------------------------------------------------
namespace {
constexpr int TI = 32, TJ = 8;

struct EoCell {
  const EoStageArgs& a;
  const int sol;
  const long cells, so;
  const int nx, ny;
  const float er, eshift, pmin_shift;
  const RKCoef rk;
  __device__ EoCell(const EoStageArgs& a_, int sol_, float dt)
      : a(a_), sol(sol_), cells((long)a_.b.x.n * a_.b.y.n), so((long)sol_ * 4 * cells), nx(a_.b.x.n), ny(a_.b.y.n),
        er(a_.eref[sol_]), eshift(a_.shift_in ? er : 0.0f), pmin_shift(a_.p_min - (a_.gamma - 1.0f) * er),
        rk(rk_coef(a_.stage, dt, a_.rk2)) {}

  // the point whose values the walls give to (J, I)
  __device__ __forceinline__ void inside(int J, int I, int& Jp, int& Ip) const {
    Jp = min(max(J, 1), ny - 2);
    Ip = min(max(I, 1), nx - 2);
  }
  // U^n with its walls (energy in the perturbation form)
  __device__ __forceinline__ void un(int J, int I, float (&u)[4]) const {
    int Jp, Ip;
    inside(J, I, Jp, Ip);
    const float* p = a.U + so + (long)Jp * nx + Ip;
#pragma unroll
    for (int c = 0; c < 4; ++c) u[c] = p[c * cells];
    u[3] -= eshift;
    if (Ip != I) u[1] = 0.0f;
    if (Jp != J) u[2] = 0.0f;
  }
  // -(dFx/dx + dFy/dy) from the products
  __device__ __forceinline__ void slope(int J, int I, float (&k)[4]) const {
    const int i = min(I, nx - 1 - I), j = min(J, ny - 1 - J);
    const float sx = (i == I) ? 0.5f : -0.5f, sy = (j == J) ? 0.5f : -0.5f;
    const long px = (long)a.nsolve * 4 * ny * a.b.ldx, py = (long)a.nsolve * 4 * a.b.y.h * nx;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const float* cx = a.b.CX + ((long)(sol * 4 + c) * ny + J) * a.b.ldx + i;
      const float* cy = a.b.CY + ((long)(sol * 4 + c) * a.b.y.h + j) * nx + I;
      // even operand -> difference of the mirror pair, odd operand -> sum
      k[c] = -((0.5f * cx[px] + sx * cx[0]) + (0.5f * cy[py] + sy * cy[0]));
    }
  }
  // stage update of one point (own products, U^n with walls, increments); ac
  // leaves with the stage's contribution and is stored by the caller, after
  // the loads of its other points
  __device__ __forceinline__ void stage(int J, int I, float (&u)[4], float (&ac)[4]) const {
    float k[4];
    un(J, I, u);
    slope(J, I, k);
    const long o = so + (long)J * nx + I;
#pragma unroll
    for (int c = 0; c < 4; ++c) ac[c] = (a.stage >= 1) ? a.acc_in[o + c * cells] : 0.0f;
#pragma unroll
    for (int c = 0; c < 4; ++c) u[c] = rk_update_incr(a.stage, rk, k[c], u[c], ac[c]);
    clamp_state<2>(u, a.gamma, a.rho_min, pmin_shift);
  }
  // the increments alone of a wall point (stages 0..2)
  __device__ __forceinline__ void wall_increment(int J, int I, float (&ac)[4]) const {
    float k[4];
    slope(J, I, k);
    const long o = so + (long)J * nx + I;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      ac[c] = (a.stage >= 1) ? a.acc_in[o + c * cells] : 0.0f;
      rk_update_incr(a.stage, rk, k[c], 0.0f, ac[c]);
    }
  }
  __device__ __forceinline__ void keep(int J, int I, const float (&ac)[4]) const {
    const long o = so + (long)J * nx + I;
#pragma unroll
    for (int c = 0; c < 4; ++c) a.acc_out[o + c * cells] = ac[c];
  }
};

// writes a row's even/odd parts of value pair (f at i, f at its mirror)
__device__ __forceinline__ void put_pair(__nv_bfloat16* dst, long plane, long parity, bool centre, float f, float fm) {
  __nv_bfloat16 q[P];
  split_parts<float>(centre ? f : f + fm, q);
#pragma unroll
  for (int p = 0; p < P; ++p) dst[p * plane] = q[p];
  split_parts<float>(centre ? 0.0f : f - fm, q);
#pragma unroll
  for (int p = 0; p < P; ++p) dst[p * plane + parity] = q[p];
}

// transposed store of a tile's even/odd y values v[c][par][side][i][j]
__device__ __forceinline__ void put_y(const EoStageArgs& a, int sol, const float* sm, int i0, int j0) {
  const int nx = a.b.x.n, hx = a.b.x.h, hy = a.b.y.h;
  const long rows = (long)a.nsolve * 4 * nx, kp = a.b.y.kp;
  const long parity = rows * kp, plane = 2 * parity;
  __nv_bfloat16* Y = static_cast<__nv_bfloat16*>(a.b.Y);
  const int j2 = 2 * (threadIdx.x & 3), il = (threadIdx.x >> 2) & 31, side = threadIdx.x >> 7;
  const int i = i0 + il, I = side ? nx - 1 - i : i;
  if (i >= hx || (side && I == i) || j0 + j2 >= hy) return;
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int par = 0; par < 2; ++par) {
      const float* v = sm + (((c * 2 + par) * 2 + side) * TI + il) * (TJ + 1) + j2;
      __nv_bfloat16 q0[P], q1[P];
      split_parts<float>(v[0], q0);
      split_parts<float>(v[1], q1);
      __nv_bfloat16* dst = Y + par * parity + ((long)(sol * 4 + c) * nx + I) * kp + j0 + j2;
#pragma unroll
      for (int p = 0; p < P; ++p)  // kp is a multiple of 8: the pad column may take the second value
        *reinterpret_cast<__nv_bfloat162*>(dst + p * plane) = __halves2bfloat162(q0[p], q1[p]);
    }
}

// stores the point's new state and the wall points that copy it
__device__ __forceinline__ void put_state(const EoStageArgs& a, const EoCell& cell, int J, int I, const float (&u)[4]) {
  if (J == 0 || I == 0 || J == cell.ny - 1 || I == cell.nx - 1) return;
  const float e = u[3] + (a.shift_out ? cell.er : 0.0f);
  auto put = [&](int j, int i) {
    float* o = a.out + cell.so + (long)j * cell.nx + i;
    o[0] = u[0];
    o[cell.cells] = (i == I) ? u[1] : 0.0f;
    o[2 * cell.cells] = (j == J) ? u[2] : 0.0f;
    o[3 * cell.cells] = e;
  };
  const int jlo = (J == 1) ? 0 : J, jhi = (J == cell.ny - 2) ? cell.ny - 1 : J;
  const int ilo = (I == 1) ? 0 : I, ihi = (I == cell.nx - 2) ? cell.nx - 1 : I;
  for (int j = jlo; j <= jhi; ++j)
    for (int i = ilo; i <= ihi; ++i) put(j, i);
}

template <int FROM, int TO>
__global__ void __launch_bounds__(TI * TJ, 2) k_eo_stage(EoStageArgs a) {
  __shared__ float sm[TO == kEoFlux ? 16 * TI * (TJ + 1) : 1];
  const int sol = blockIdx.z;
  dep_wait();
  if (a.active != nullptr && a.active[sol] == 0) return;
  const float dt = (a.dt_dev != nullptr) ? (float)a.dt_dev[sol] : (float)a.dt;
  const EoCell cell(a, sol, dt);
  const int nx = cell.nx, ny = cell.ny, hx = a.b.x.h, hy = a.b.y.h;
  const int il = threadIdx.x % TI, jl = threadIdx.x / TI;
  const int i0 = blockIdx.x * TI, j0 = blockIdx.y * TJ;
  const int i = i0 + il, j = j0 + jl;
  const bool in = i < hx && j < hy;
  const int im = nx - 1 - i, jm = ny - 1 - j;
  const bool ci = im == i, cj = jm == j;  // centre line / row: its own mirror
  float u[4][4] = {}, ac[4][4];  // points (j, i), (j, im), (jm, i), (jm, im)
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    const int J = (p & 2) ? jm : j, I = (p & 1) ? im : i;
    if (!in) {
#pragma unroll
      for (int c = 0; c < 4; ++c) u[p][c] = 1.0f;
    } else if (FROM == kEoStart) {
      cell.un(J, I, u[p]);
    } else {
      // a launch that writes the state skips the walls: their U^n may be in the making
      const bool wall = i == 0 || j == 0;
      if (TO == kEoOut && wall) continue;
      if (TO == kEoFlux) {
        // a wall point takes its interior neighbour's new state; its own
        // increments are kept only for the filter, which sees the raw walls
        int Jp, Ip;
        cell.inside(J, I, Jp, Ip);
        cell.stage(Jp, Ip, u[p], ac[p]);
        if (wall) {
          if (Ip != I) u[p][1] = 0.0f;
          if (Jp != J) u[p][2] = 0.0f;
          if (a.wall_acc) cell.wall_increment(J, I, ac[p]);
        }
      } else {
        cell.stage(J, I, u[p], ac[p]);
      }
    }
  }
  if constexpr (FROM == kEoStage && TO == kEoFlux) {
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      const bool dup = ((p & 1) && ci) || ((p & 2) && cj);
      if (in && !dup && (a.wall_acc || (i > 0 && j > 0))) cell.keep((p & 2) ? jm : j, (p & 1) ? im : i, ac[p]);
    }
  }
  if constexpr (TO == kEoOut) {
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      const int J = (p & 2) ? jm : j, I = (p & 1) ? im : i;
      const bool dup = ((p & 1) && ci) || ((p & 2) && cj);
      if (in && !dup) put_state(a, cell, J, I, u[p]);
    }
    return;
  }
  const long rowsX = (long)a.nsolve * 4 * ny;
  const long parX = rowsX * a.b.x.kp, planeX = 2 * parX;
  __nv_bfloat16* X = static_cast<__nv_bfloat16*>(a.b.X);
  if constexpr (TO == kEoFilterX) {
    // complement C = I - F of the filter on rows relative to their first value
    // (F keeps constants); the new state goes to S for V = S - C S
#pragma unroll 1
    for (int q = 0; q < 2; ++q) {
      const int J = q ? jm : j;
      if (!in || (q && cj)) break;
      float f0[4];
      float f1[4];
      cell.stage(J, 0, f0, f1);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float f = q ? u[2][c] : u[0][c], fm = q ? u[3][c] : u[1][c];
        put_pair(X + ((long)(sol * 4 + c) * ny + J) * a.b.x.kp + i, planeX, parX, ci, f - f0[c], fm - f0[c]);
        float* S = a.S + cell.so + c * cell.cells + (long)J * nx;
        S[i] = f;
        S[im] = fm;
      }
    }
    return;
  }
  if constexpr (TO == kEoFlux) {
    const float gm1 = a.gamma - 1.0f, geref = a.gamma * cell.er;
    float fx[4][4], fy[4][4];
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      const float rho = u[p][0], mx = u[p][1], my = u[p][2], e = u[p][3];
      const float ux = mx / rho, uy = my / rho;
      const float pp = gm1 * (e - 0.5f * rho * (ux * ux + uy * uy));
      const float hh = e + pp + geref;
      fx[p][0] = rho * ux;
      fx[p][1] = rho * ux * ux + pp;
      fx[p][2] = rho * uy * ux;
      fx[p][3] = hh * ux;
      fy[p][0] = rho * uy;
      fy[p][1] = rho * ux * uy;
      fy[p][2] = rho * uy * uy + pp;
      fy[p][3] = hh * uy;
    }
    if (in) {
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        put_pair(X + ((long)(sol * 4 + c) * ny + j) * a.b.x.kp + i, planeX, parX, ci, fx[0][c], fx[1][c]);
        if (!cj) put_pair(X + ((long)(sol * 4 + c) * ny + jm) * a.b.x.kp + i, planeX, parX, ci, fx[2][c], fx[3][c]);
      }
    }
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int side = 0; side < 2; ++side) {
        const float f = fy[side][c], fm = fy[2 + side][c];
        sm[(((c * 2 + 0) * 2 + side) * TI + il) * (TJ + 1) + jl] = cj ? f : f + fm;
        sm[(((c * 2 + 1) * 2 + side) * TI + il) * (TJ + 1) + jl] = cj ? 0.0f : f - fm;
      }
    __syncthreads();
    put_y(a, sol, sm, i0, j0);
  }
}

// state after the x filter at (J, I): S - C_x S from the products
__device__ __forceinline__ void x_filtered(const EoStageArgs& a, int sol, int J, int I, float (&v)[4]) {
  const int nx = a.b.x.n, ny = a.b.y.n, i = min(I, nx - 1 - I);
  const float sx = (i == nx - 1 - i) ? 0.0f : (i == I) ? 0.5f : -0.5f;  // (a centre's difference is zero)
  const long px = (long)a.nsolve * 4 * ny * a.b.ldx, cells = (long)nx * ny;
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const float* cx = a.b.CX + ((long)(sol * 4 + c) * ny + J) * a.b.ldx + i;
    v[c] = a.S[((long)sol * 4 + c) * cells + (long)J * nx + I] - (0.5f * cx[0] + sx * cx[px]);
  }
}

__global__ void __launch_bounds__(TI * TJ) k_eo_filter_y(EoStageArgs a) {
  __shared__ float sm[16 * TI * (TJ + 1)];
  const int sol = blockIdx.z;
  dep_wait();
  if (a.active != nullptr && a.active[sol] == 0) return;
  const int nx = a.b.x.n, ny = a.b.y.n, hx = a.b.x.h, hy = a.b.y.h;
  const int il = threadIdx.x % TI, jl = threadIdx.x / TI;
  const int i0 = blockIdx.x * TI, j0 = blockIdx.y * TJ;
  const int i = i0 + il, j = j0 + jl, jm = ny - 1 - j;
  const bool in = i < hx && j < hy, cj = jm == j;
#pragma unroll
  for (int side = 0; side < 2; ++side) {
    const int I = side ? nx - 1 - i : i;
    float f[4] = {0.f, 0.f, 0.f, 0.f}, fm[4] = {0.f, 0.f, 0.f, 0.f};
    if (in) {
      float f0[4];
      x_filtered(a, sol, 0, I, f0);
      x_filtered(a, sol, j, I, f);
      x_filtered(a, sol, jm, I, fm);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        float* V = a.V + ((long)sol * 4 + c) * nx * ny + I;
        V[(long)j * nx] = f[c];
        V[(long)jm * nx] = fm[c];
        f[c] -= f0[c];
        fm[c] -= f0[c];
      }
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      sm[(((c * 2 + 0) * 2 + side) * TI + il) * (TJ + 1) + jl] = cj ? f[c] : f[c] + fm[c];
      sm[(((c * 2 + 1) * 2 + side) * TI + il) * (TJ + 1) + jl] = cj ? 0.0f : f[c] - fm[c];
    }
  }
  __syncthreads();
  put_y(a, sol, sm, i0, j0);
}

__global__ void __launch_bounds__(TI * TJ) k_eo_filter_out(EoStageArgs a) {
  const int sol = blockIdx.z;
  dep_wait();
  if (a.active != nullptr && a.active[sol] == 0) return;
  const EoCell cell(a, sol, 0.0f);
  const int nx = cell.nx, ny = cell.ny, hy = a.b.y.h;
  const int I = blockIdx.x * TI + threadIdx.x % TI, J = blockIdx.y * TJ + threadIdx.x / TI;
  if (I >= nx || J >= ny) return;
  const int j = min(J, ny - 1 - J);
  const float sy = (j == ny - 1 - j) ? 0.0f : (j == J) ? 0.5f : -0.5f;
  const long py = (long)a.nsolve * 4 * hy * nx;
  float u[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const float* cy = a.b.CY + ((long)(sol * 4 + c) * hy + j) * nx + I;
    u[c] = a.V[cell.so + c * cell.cells + (long)J * nx + I] - (0.5f * cy[0] + sy * cy[py]);
  }
  put_state(a, cell, J, I, u);
}

dim3 eo_grid(const EoStageArgs& a) {
  return dim3((a.b.x.h + TI - 1) / TI, (a.b.y.h + TJ - 1) / TJ, a.nsolve);
}
cudaError_t eo_stage_any(const EoStageArgs& a, int from, int to, cudaStream_t s) {
  const dim3 g = eo_grid(a);
  if (from == kEoStart && to == kEoFlux) return launch_dep(k_eo_stage<kEoStart, kEoFlux>, g, TI * TJ, 0, s, a);
  if (from == kEoStage && to == kEoFlux) return launch_dep(k_eo_stage<kEoStage, kEoFlux>, g, TI * TJ, 0, s, a);
  if (from == kEoStage && to == kEoFilterX) return launch_dep(k_eo_stage<kEoStage, kEoFilterX>, g, TI * TJ, 0, s, a);
  if (from == kEoStage && to == kEoOut) return launch_dep(k_eo_stage<kEoStage, kEoOut>, g, TI * TJ, 0, s, a);
  return cudaErrorInvalidValue;
}
}  // namespace

cudaError_t launch_eo_stage(const EoStageArgs& a, int from, int to, cudaStream_t s) {
  return eo_stage_any(a, from, to, s);
}
cudaError_t launch_eo_filter_y(const EoStageArgs& a, cudaStream_t s) {
  return launch_dep(k_eo_filter_y, eo_grid(a), TI * TJ, 0, s, a);
}
cudaError_t launch_eo_filter_out(const EoStageArgs& a, cudaStream_t s) {
  return launch_dep(k_eo_filter_out, dim3((a.b.x.n + TI - 1) / TI, (a.b.y.n + TJ - 1) / TJ, a.nsolve), TI * TJ, 0, s, a);
}

}  // namespace ps

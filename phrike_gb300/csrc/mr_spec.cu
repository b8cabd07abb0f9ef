// Truncated-spectra passes for 5-smooth axes (see mr_spec.cuh).
#include <cuda_runtime.h>
#include <limits.h>
#include <math.h>

#include <algorithm>
#include <vector>

#include "launch.cuh"
#include "mr_fft.cuh"
#include "mr_spec.cuh"

namespace ps {
namespace {

using mrfft::qdiv;

constexpr int kThreads = 512;
constexpr int kWide = 768;  // strided passes (80 registers)

// ---------------------------------------------------------------- transforms
template <int R, bool INV>
__device__ __forceinline__ void rdft(float2 (&v)[R]) {
  if constexpr (R == 2 || R == 3 || R == 4 || R == 5) {
    mrfft::dft_small<R>(v, INV);
  } else if constexpr (R == 8 || R == 16) {
    dft<R, INV>(v);
  } else {  // R = R1 R2: n = R2 n1 + n2, k = k1 + R1 k2
    constexpr int R1 = (R % 3 == 0) ? 3 : 2, R2 = R / R1;
    float2 y[R1][R2];
    sfor<0, R2>([&](auto n2c) {
      constexpr int n2 = decltype(n2c)::value;
      float2 x[R1];
      sfor<0, R1>([&](auto n1c) { x[decltype(n1c)::value] = v[R2 * decltype(n1c)::value + n2]; });
      mrfft::dft_small<R1>(x, INV);
      sfor<0, R1>([&](auto kc) {
        constexpr int k1 = decltype(kc)::value;
        y[k1][n2] = twmul<R, k1 * n2, INV>(x[k1]);
      });
    });
    sfor<0, R1>([&](auto kc) {
      constexpr int k1 = decltype(kc)::value;
      mrfft::dft_small<R2>(y[k1], INV);
      sfor<0, R2>([&](auto k2c) { v[k1 + R1 * decltype(k2c)::value] = y[k1][decltype(k2c)::value]; });
    });
  }
}

// Signals of a CTA in shared memory.  ROWS: nsig pencils one after the other;
// else nsig tiles [element][T], T a power of two.
struct Lay {
  float2* buf;
  int stride;   // float2 between signals
  int nsig;
  int lt;       // log2 T (strided)
};

// Element of point i (digits from the first pass down) and of mode k after the
// forward passes (digits from the first pass up).
__device__ __forceinline__ int elem_of_point(const SpecAxis& ax, int i) {
  int e = 0;
  for (int s = 0; s < ax.nst - 1; ++s) {
    const int q = qdiv(i, ax.inv_m[s]);
    i -= q * ax.m[s];
    e += q * ax.st[s];
  }
  return e + i;
}
__device__ __forceinline__ int elem_of_mode(const SpecAxis& ax, int k) {
  int e = 0;
  for (int s = 0; s < ax.nst - 1; ++s) {
    const int t = qdiv(k, ax.inv_r[s]);
    e += (k - t * ax.radix[s]) * ax.st[s];
    k = t;
  }
  return e + k;
}

// A pass of radix R over blocks of length L: butterflies over its digit, in
// place.  A thread keeps one butterfly index j for all the signals it serves
// (its address is found once); with more threads than butterflies
// the signals are dealt out over groups of n/R threads.
template <int R, bool INV, bool ROWS>
__device__ __forceinline__ void pass(const Lay& g, const SpecAxis& ax, const float2* tw, int L, int step) {
  const int m = L / R, nb = ax.n / R;
  tw += ax.n - L;
  const float im = 1.0f / (float)m;
  const int lt = ROWS ? 0 : g.lt;
  const int W = blockDim.x >> lt;
  const int u = threadIdx.x >> lt, col = ROWS ? 0 : threadIdx.x & ((1 << lt) - 1);
  step <<= lt;
  int slots = 1, s0 = 0, j = u;
  if (W >= 2 * nb) {
    slots = W / nb;
    s0 = qdiv(u, 1.0f / (float)nb);
    j = u - s0 * nb;
    if (s0 >= slots) return;
  }
#pragma unroll 1
  for (; j < nb; j += W) {
    const int b = qdiv(j, im), i = j - b * m;
    const int e0 = elem_of_point(ax, b * L + i);
    const float2* w = tw + i;
    float2* p = g.buf + ((ROWS ? e0 : (e0 << lt)) + col) + s0 * g.stride;
#pragma unroll 1
    for (int s = s0; s < g.nsig; s += slots, p += slots * g.stride) {
      float2 v[R];
#pragma unroll
      for (int q = 0; q < R; ++q) v[q] = p[q * step];
      if (INV && m > 1) {
#pragma unroll
        for (int q = 1; q < R; ++q) v[q] = ps::cmulc(v[q], w[(q - 1) * m]);
      }
      rdft<R, INV>(v);
      if (!INV && m > 1) {
#pragma unroll
        for (int q = 1; q < R; ++q) v[q] = ps::cmul(v[q], w[(q - 1) * m]);
      }
#pragma unroll
      for (int q = 0; q < R; ++q) p[q * step] = v[q];
    }
    if (slots > 1) break;
  }
}

template <bool INV, bool ROWS>
__device__ __forceinline__ void pass_any(int R, const Lay& g, const SpecAxis& ax, const float2* tw, int L, int step) {
  switch (R) {
#define PS_R(K) \
  case K:       \
    pass<K, INV, ROWS>(g, ax, tw, L, step); \
    break;
    PS_R(2)
    PS_R(3)
    PS_R(4)
    PS_R(5)
    PS_R(6)
    PS_R(8)
    PS_R(9)
    PS_R(10)
    PS_R(12)
    PS_R(15)
    PS_R(16)
#undef PS_R
    default:
      break;
  }
}

// All threads call; the buffers are complete on entry (a barrier first) and
// on return.
template <bool ROWS>
__device__ __forceinline__ void forward(const Lay& g, const SpecAxis& ax, const float2* tw) {
  __syncthreads();
  int L = ax.n;
#pragma unroll 1
  for (int s = 0; s < ax.nst; ++s) {
    const int R = ax.radix[s];
    pass_any<false, ROWS>(R, g, ax, tw, L, ax.st[s]);
    __syncthreads();
    L /= R;
  }
}
template <bool ROWS>
__device__ __forceinline__ void inverse(const Lay& g, const SpecAxis& ax, const float2* tw) {
  __syncthreads();
  int L = 1;
#pragma unroll 1
  for (int s = ax.nst - 1; s >= 0; --s) {
    const int R = ax.radix[s];
    L *= R;
    pass_any<true, ROWS>(R, g, ax, tw, L, ax.st[s]);
    __syncthreads();
  }
}

// 8-byte asynchronous copy, zero unless take
__device__ __forceinline__ void cp8(void* dst, const void* src, bool take) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(smem_addr(dst)), "l"(src), "r"(take ? 8 : 0)
               : "memory");
}

__device__ __forceinline__ void cp4(void* dst, const void* src, bool take) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_addr(dst)), "l"(src), "r"(take ? 4 : 0)
               : "memory");
}

// The axis' tables in shared memory: twiddles, then P and d (4 n words).
struct Tables {
  const float2* tw;
  const float* P;
  const float* d;
};

// Starts the copies (the caller commits and waits before forward / inverse).
__device__ __forceinline__ Tables load_tables(float2* at, const SpecAxis& ax) {
  const int n = ax.n;
  float* P = reinterpret_cast<float*>(at + n);
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    cp8(at + i, ax.tw + i, true);
    cp4(P + i, ax.P + i, true);
    cp4(P + n + i, ax.d + i, true);
  }
  return Tables{at, P, P + n};
}
// mode of column m, and column of mode k (-1: masked)
__device__ __forceinline__ int mode_of(const SpecAxis& ax, int m) { return m <= ax.km ? m : m + ax.n - 2 * ax.km - 1; }
__device__ __forceinline__ int col_of(const SpecAxis& ax, int k) {
  return k <= ax.km ? k : (k >= ax.n - ax.km ? k - (ax.n - 2 * ax.km - 1) : -1);
}

// ---------------------------------------------------------------- x rows
// One CTA: `pg` rows.  2D transforms all flux pairs of a row together; 3D
// keeps the primitives in shared memory and takes one direction at a time.
template <int ND, bool INC, bool FLUX>
__global__ void __launch_bounds__(kThreads, 1) k_mrs_x(SpecXArgs a, SpecAxis ax, int pg) {
  constexpr int NC = ND + 2, NP = NC / 2;
  constexpr bool ODD = (NC % 2) != 0;
  constexpr int NJ = NP + (ODD ? 1 : 0);
  constexpr int DIRS = (ND == 2) ? 2 : 1;  // directions transformed together
  extern __shared__ __align__(16) float2 sm[];
  __shared__ float red[32];
  const int n = ax.n, M = 2 * ax.km + 1, stride = ax.len;
  const int nsig = (FLUX ? DIRS : 1) * NJ;
  float2* buf = sm + 2 * n;                                                // [nsig][pg][stride]
  float* prim = reinterpret_cast<float*>(buf + (long)nsig * pg * stride);  // 3D fluxes: [NC][pg][n]
  const int row0 = blockIdx.x * pg;
  const Tables tb = load_tables(sm, ax);
  cp_commit();
  dep_wait();
  // rows of a CTA belong to one solve (rps is a multiple of pg, or pg = 1)
  const int sol = row0 / a.rps;
  if (a.active != nullptr && a.active[sol] == 0) {
    cp_wait<0>();
    return;
  }
  const float inv_n = 1.0f / (float)n;
  const float er = a.eref[sol];
  const float eshift = a.shift_in ? er : 0.0f;
  const float g1 = a.gamma - 1.0f, ig1 = 1.0f / g1;
  const float pref = g1 * er, href = a.gamma * er;
  const float pmin_shift = a.p_min - pref;

  if constexpr (INC) {
    // spectra of the increment into digit-reversed places, zero where masked
#pragma unroll 2
    for (int e = threadIdx.x; e < pg * n; e += blockDim.x) {
      const int r = qdiv(e, inv_n), k = e - r * n;
      const int m = col_of(ax, k);
      const float2* d = a.D + (long)(row0 + r) * a.pitch;
      float2* to = buf + r * stride + elem_of_mode(ax, k);
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        if (ODD && j == NP && m > ax.km) {  // half spectra: X(-k) = conj X(k)
          const float2 v = d[j * M + n - k];
          to[j * pg * stride] = make_float2(v.x, -v.y);
        } else {
          cp8(to + j * pg * stride, m >= 0 ? d + j * M + m : d, m >= 0);
        }
      }
    }
    cp_commit();
    cp_wait<0>();
    inverse<true>(Lay{buf, stride, NJ * pg, 0}, ax, tb.tw);
  } else {
    cp_wait<0>();
    __syncthreads();
  }

  float smax = 0.0f;
  const long ubase = (long)sol * a.ssU + (long)(row0 % a.rps) * n;
  const int tot = pg * n;
  constexpr int UB = 4;  // points whose loads are issued together
  for (int e0 = threadIdx.x; e0 < tot; e0 += UB * blockDim.x) {
    float ub[UB][NC];
#pragma unroll
    for (int h = 0; h < UB; ++h) {
      const int e = e0 + h * blockDim.x;
#pragma unroll
      for (int c = 0; c < NC; ++c) ub[h][c] = (e < tot) ? a.U[ubase + c * a.fs + e] : 1.0f;
    }
#pragma unroll
   for (int h = 0; h < UB; ++h) {
    const int e = e0 + h * blockDim.x;
    if (e >= tot) break;
    const int r = qdiv(e, inv_n), i = e - r * n;
    const int at = r * stride + elem_of_point(ax, i);
    float u[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) u[c] = ub[h][c];
    u[NC - 1] -= eshift;
    if constexpr (INC) {
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        const float2 v = buf[j * pg * stride + at];
        u[2 * j] += v.x;
        if (2 * j + 1 < NC) u[2 * j + 1 < NC ? 2 * j + 1 : 0] += v.y;
      }
      if constexpr (ND == 2) clamp_state<ND>(u, a.gamma, a.rho_min, pmin_shift);
      if (a.Uw != nullptr) {
#pragma unroll
        for (int c = 0; c < NC; ++c)
          a.Uw[ubase + c * a.fs + e] = u[c] + ((c == NC - 1 && a.shift_out) ? er : 0.0f);
      }
    }
    if constexpr (FLUX) {
      const float rho = u[0], rinv = 1.0f / rho;
      float vel[ND], kin = 0.0f;
#pragma unroll
      for (int d = 0; d < ND; ++d) {
        vel[d] = u[1 + d] * rinv;
        kin = fmaf(vel[d], vel[d], kin);
      }
      const float pr = g1 * (u[NC - 1] - 0.5f * rho * kin);
      if (a.speed != nullptr) {
        const float cs = sqrtf(a.gamma * (pr + pref) * rinv);
        float um = fabsf(vel[0]);
        if (ND == 3) um = fmaxf(um, fmaxf(fabsf(vel[1]), fabsf(vel[ND - 1])));
        smax = fmaxf(smax, um + cs);
      }
      if constexpr (ND == 2) {
        const float ept = (fmaf(pr, ig1, 0.5f * rho * kin) + pr) + href;
#pragma unroll
        for (int d = 0; d < 2; ++d) {
          const float mn = rho * vel[d];
          buf[(d * NJ + 0) * pg * stride + at] = make_float2(mn, mn * vel[0] + (d == 0 ? pr : 0.0f));
          buf[(d * NJ + 1) * pg * stride + at] = make_float2(mn * vel[1] + (d == 1 ? pr : 0.0f), ept * vel[d]);
        }
      } else {
        prim[e] = rho;
#pragma unroll
        for (int d = 0; d < ND; ++d) prim[(1 + d) * tot + e] = vel[d];
        prim[(NC - 1) * tot + e] = pr;
      }
    }
   }
  }
  if constexpr (FLUX) {
    if (a.speed != nullptr) {
      const float m = block_max(smax, red);
      if (threadIdx.x == 0) atomic_max_nonneg(a.speed + sol, m);
    }
    for (int d0 = 0; d0 < ND; d0 += DIRS) {
      if constexpr (ND == 3) {
        __syncthreads();
        for (int e = threadIdx.x; e < tot; e += blockDim.x) {
          const int r = qdiv(e, inv_n), i = e - r * n;
          const int at = r * stride + elem_of_point(ax, i);
          const float rho = prim[e], ux = prim[tot + e], uy = prim[2 * tot + e], uz = prim[3 * tot + e];
          const float pr = prim[4 * tot + e];
          const float un = d0 == 0 ? ux : d0 == 1 ? uy : uz;
          const float mn = rho * un;
          const float kin = fmaf(uz, uz, fmaf(uy, uy, ux * ux));
          const float ept = (fmaf(pr, ig1, 0.5f * rho * kin) + pr) + href;
          buf[at] = make_float2(mn, mn * ux + (d0 == 0 ? pr : 0.0f));
          buf[pg * stride + at] = make_float2(mn * uy + (d0 == 1 ? pr : 0.0f), mn * uz + (d0 == 2 ? pr : 0.0f));
          buf[2 * pg * stride + at] = make_float2(ept * un, 0.0f);
        }
      }
      forward<true>(Lay{buf, stride, DIRS * NJ * pg, 0}, ax, tb.tw);
      // kept modes, in order: D along x for direction 0, P else
      const float inv_m = 1.0f / (float)M;
#pragma unroll 2
      for (int e = threadIdx.x; e < pg * M; e += blockDim.x) {
        const int r = qdiv(e, inv_m), m = e - r * M;
        const int k = mode_of(ax, m);
        const float2* from = buf + r * stride + elem_of_mode(ax, k);
        const float P = tb.P[k], dd = tb.d[k];
        float2* to = a.G + (long)(row0 + r) * a.pitch + m;
#pragma unroll
        for (int dj = 0; dj < DIRS * NJ; ++dj) {
          const int dir = d0 + dj / NJ, j = dj % NJ;
          if (ODD && j == NP && m > ax.km) continue;
          const float2 v = from[dj * pg * stride];
          to[dir * a.gs + j * M] = (dir == 0) ? make_float2(-v.y * dd, v.x * dd) : make_float2(v.x * P, v.y * P);
        }
      }
    }
  }
}

// ---------------------------------------------------------------- strided
// One CTA per tile of columns and outer index (plane, or solve and outer line),
// tiles fastest, all in gridDim.x: planes times solves pass the 65535 of gridDim.y.
__device__ __forceinline__ int outer_of(int ncol, int lt, int* col0) {
  const int tiles = (ncol + (1 << lt) - 1) >> lt;
  const int o = blockIdx.x / tiles;
  *col0 = (blockIdx.x - o * tiles) << lt;
  return o;
}

// rows x T tile -> shared memory, row i at element at[i], 16 bytes at a time
template <typename At>
__device__ __forceinline__ void tile_in(float2* dst, int lt, int rows, const float2* src, long as, int col0, int ncol,
                                        At&& at) {
  const int lc = lt - 1;
#pragma unroll 4
  for (int e = threadIdx.x; e < rows << lc; e += blockDim.x) {
    const int i = e >> lc, c = 2 * (e & ((1 << lc) - 1));
    const bool take = col0 + c < ncol;
    cp16(dst + (at(i) << lt) + c, take ? src + i * as + col0 + c : src, take);
  }
}

template <int MAXT>
__global__ void __launch_bounds__(MAXT, 1) k_mrs_f(SpecFArgs a, SpecAxis ax, int lt) {
  extern __shared__ __align__(16) float2 sm[];
  const int T = 1 << lt, n = ax.n, M = 2 * ax.km + 1;
  const int stride = ax.len << lt;
  float2* buf = sm;
  int col0;
  const int plane = outer_of(a.ncol, lt, &col0);
  const Tables tb = load_tables(buf + 2 * stride, ax);
  dep_wait();
  if (a.active != nullptr && a.active[plane / a.pps] == 0) {
    cp_wait<0>();
    return;
  }
  const float2* in = a.G + (long)plane * n * a.pitch;
  auto same = [&](int i) { return elem_of_point(ax, i); };
  tile_in(buf, lt, n, in, a.pitch, col0, a.ncol, same);
  tile_in(buf + stride, lt, n, in + a.gs, a.pitch, col0, a.ncol, same);
  cp_commit();
  cp_wait<0>();
  forward<false>(Lay{buf, stride, 2, lt}, ax, tb.tw);
  float2* out = a.out + (long)plane * M * a.pitch;
#pragma unroll 4
  for (int e = threadIdx.x; e < M << lt; e += blockDim.x) {
    const int m = e >> lt, c = e & (T - 1), k = mode_of(ax, m);
    const int at = (elem_of_mode(ax, k) << lt) + c;
    const float P = tb.P[k], d = tb.d[k];
    const float2 v = buf[at], z = buf[stride + at];
    if (col0 + c < a.ncol)
      out[(long)m * a.pitch + col0 + c] = make_float2(fmaf(P, v.x, -d * z.y), fmaf(P, v.y, d * z.x));
  }
  __syncthreads();
  tile_in(buf, lt, n, in + 2 * a.gs, a.pitch, col0, a.ncol, same);
  cp_commit();
  cp_wait<0>();
  forward<false>(Lay{buf, stride, 1, lt}, ax, tb.tw);
  out += a.os;
#pragma unroll 4
  for (int e = threadIdx.x; e < M << lt; e += blockDim.x) {
    const int m = e >> lt, c = e & (T - 1), k = mode_of(ax, m);
    const float P = tb.P[k];
    const float2 v = buf[(elem_of_mode(ax, k) << lt) + c];
    if (col0 + c < a.ncol) out[(long)m * a.pitch + col0 + c] = make_float2(P * v.x, P * v.y);
  }
}

template <int MAXT>
__global__ void __launch_bounds__(MAXT, 1) k_mrs_c(SpecCArgs a, SpecAxis ax, int lt) {
  extern __shared__ __align__(16) float2 sm[];
  const int T = 1 << lt, n = ax.n;
  const int stride = ax.len << lt;
  float2* buf = sm;
  int col0;
  const int o = outer_of(a.ncol, lt, &col0), outer = o % a.nouter, sol = o / a.nouter;
  const Tables tb = load_tables(buf + 2 * stride, ax);
  dep_wait();
  if (a.active != nullptr && a.active[sol] == 0) {
    cp_wait<0>();
    return;
  }
  const long base = (long)sol * a.ss + (long)outer * a.os;
  auto same = [&](int i) { return elem_of_point(ax, i); };
  tile_in(buf, lt, n, a.a + base, a.as, col0, a.ncol, same);
  tile_in(buf + stride, lt, n, a.b + base, a.as, col0, a.ncol, same);
  cp_commit();
  const float dt = (a.dt_dev != nullptr) ? (float)a.dt_dev[sol] : (float)a.dt;
  const RKCoef rk = rk_coef(a.stage, dt, a.rk2);
  cp_wait<0>();
  forward<false>(Lay{buf, stride, 2, lt}, ax, tb.tw);
  float2* acc = a.acc + (long)sol * a.acc_ss + (long)outer * a.acc_os + col0;
  constexpr int UB = 4;  // accumulator loads issued together
  for (int e0 = threadIdx.x; e0 < n << lt; e0 += UB * blockDim.x) {
    float2 qa[UB];
#pragma unroll
    for (int h = 0; h < UB; ++h) {
      const int e = e0 + h * blockDim.x, k = e >> lt, c = e & (T - 1);
      const int m = k < n ? col_of(ax, k) : -1;
      qa[h] = make_float2(0.0f, 0.0f);
      if (a.stage != 0 && m >= 0 && col0 + c < a.ncol) qa[h] = acc[m * a.acc_as + c];
    }
#pragma unroll
    for (int h = 0; h < UB; ++h) {
      const int e = e0 + h * blockDim.x, k = e >> lt, c = e & (T - 1);
      if (k >= n) break;
      const int at = (elem_of_mode(ax, k) << lt) + c;
      const int m = col_of(ax, k);
      float2 inc = make_float2(0.0f, 0.0f);
      if (m >= 0) {
        const float P = -tb.P[k], d = -tb.d[k];
        const float2 v = buf[at], z = buf[stride + at];
        const float2 kk = make_float2(fmaf(P, v.x, -d * z.y), fmaf(P, v.y, d * z.x));
        const float2 q = make_float2(fmaf(rk.wacc, kk.x, qa[h].x), fmaf(rk.wacc, kk.y, qa[h].y));
        if (a.stage == 3) {
          inc = q;
        } else {
          if (col0 + c < a.ncol) acc[m * a.acc_as + c] = q;
          inc = make_float2(rk.wnext * kk.x, rk.wnext * kk.y);
        }
      }
      buf[at] = inc;
    }
  }
  inverse<false>(Lay{buf, stride, 1, lt}, ax, tb.tw);
  float2* out = a.out + base + col0;
#pragma unroll 4
  for (int e = threadIdx.x; e < n << lt; e += blockDim.x) {
    const int i = e >> lt, c = e & (T - 1);
    if (col0 + c < a.ncol) out[i * a.as + c] = buf[(elem_of_point(ax, i) << lt) + c];
  }
}

template <int MAXT>
__global__ void __launch_bounds__(MAXT, 1) k_mrs_i(SpecIArgs a, SpecAxis ax, int lt) {
  extern __shared__ __align__(16) float2 sm[];
  const int T = 1 << lt, n = ax.n, M = 2 * ax.km + 1;
  float2* buf = sm;
  int col0;
  const int plane = outer_of(a.ncol, lt, &col0);
  const Tables tb = load_tables(buf + (ax.len << lt), ax);
  dep_wait();
  if (a.active != nullptr && a.active[plane / a.pps] == 0) {
    cp_wait<0>();
    return;
  }
  tile_in(buf, lt, M, a.in + (long)plane * M * a.pitch, a.pitch, col0, a.ncol,
          [&](int m) { return elem_of_mode(ax, mode_of(ax, m)); });
  cp_commit();
  for (int e = threadIdx.x; e < (n - M) << lt; e += blockDim.x)  // masked modes
    buf[(elem_of_mode(ax, ax.km + 1 + (e >> lt)) << lt) + (e & (T - 1))] = make_float2(0.0f, 0.0f);
  cp_wait<0>();
  inverse<false>(Lay{buf, 0, 1, lt}, ax, tb.tw);
  float2* out = a.D + (long)plane * n * a.pitch + col0;
#pragma unroll 4
  for (int e = threadIdx.x; e < n << lt; e += blockDim.x) {
    const int i = e >> lt, c = e & (T - 1);
    if (col0 + c < a.ncol) out[(long)i * a.pitch + c] = buf[(elem_of_point(ax, i) << lt) + c];
  }
}

// ---------------------------------------------------------------- filter
// Complementary filter along one axis, pairs of real fields in one complex
// signal.  ROWS (x): T pencils of one solve per CTA; strided: T adjacent pencils.
// PER: CTAs per SM that the registers are cut for.
template <bool ROWS, int PER>
__global__ void __launch_bounds__(kThreads, PER) k_mrs_filter(MrFilterArgs a, SpecAxis ax, int lt) {
  extern __shared__ __align__(16) float2 sm[];
  const int n = ax.n, T = 1 << lt;
  const int stride = ROWS ? ax.len : ax.len << lt;
  float2* buf = sm + 2 * n;
  const int sol = blockIdx.y;
  const Tables tb = load_tables(sm, ax);
  dep_wait();
  if (a.active != nullptr && a.active[sol] == 0) {
    cp_wait<0>();
    return;
  }
  const long j0 = (long)blockIdx.x * T;  // first pencil
  const float inv_n = 1.0f / (float)n;
  const int fa = 2 * blockIdx.z;         // field pair of this CTA
  const bool two = fa + 1 < a.nf;
  const float* in = a.in + (long)sol * a.ss_in + fa * a.fs;
  float* out = a.out + (long)sol * a.ss_out + fa * a.fs;
  // strided: a thread keeps its pencil (the block is a multiple of T wide)
  const int q0 = threadIdx.x & (T - 1);
  const bool v0 = j0 + q0 < a.npen;
  const long b0 = ROWS ? j0 * n : (v0 ? ((j0 + q0) / a.es) * a.es * n + (j0 + q0) % a.es : 0);
  const int left = (int)((a.npen - j0 < T ? a.npen - j0 : T) * n);  // rows: elements of valid pencils
  auto each = [&](auto&& f) {  // f(element, offset, valid)
#pragma unroll 4
    for (int e = threadIdx.x; e < n << lt; e += blockDim.x) {
      if (ROWS) {
        const int q = qdiv(e, inv_n), i = e - q * n;
        f(q * stride + elem_of_point(ax, i), b0 + e, e < left);
      } else {
        const int i = e >> lt;
        f((elem_of_point(ax, i) << lt) + q0, b0 + (long)i * a.es, v0);
      }
    }
  };
  each([&](int at, long off, bool valid) {  // (4-byte asynchronous copies: all loads in flight)
    cp4(&buf[at].x, valid ? in + off : in, valid);
    cp4(&buf[at].y, valid && two ? in + a.fs + off : in, valid && two);
  });
  cp_commit();
  cp_wait<0>();
  const Lay g{buf, stride, ROWS ? T : 1, ROWS ? 0 : lt};
  forward<ROWS>(g, ax, tb.tw);
  for (int e = threadIdx.x; e < n << lt; e += blockDim.x) {
    const int q = ROWS ? qdiv(e, inv_n) : q0, k = ROWS ? e - q * n : e >> lt;
    const int p = elem_of_mode(ax, k);
    const float s = (1.0f / n) - tb.P[k];
    float2& w = buf[ROWS ? q * stride + p : (p << lt) + q];
    w = make_float2(w.x * s, w.y * s);
  }
  inverse<ROWS>(g, ax, tb.tw);
  const bool last = a.eadd != nullptr && fa + 2 >= a.nf;
  const float ea = (last && !two) ? a.eadd[sol] : 0.0f, eb = (last && two) ? a.eadd[sol] : 0.0f;
  // the fields once more (L2), eight points' loads together
  constexpr int UB = 8;
  for (int e0 = threadIdx.x; e0 < n << lt; e0 += UB * blockDim.x) {
    float2 x[UB];
    long off[UB];
    int at[UB];
#pragma unroll
    for (int h = 0; h < UB; ++h) {
      const int e = e0 + h * blockDim.x;
      bool valid = e < n << lt;
      if (ROWS) {
        const int q = qdiv(e, inv_n), i = e - q * n;
        valid = e < left;
        at[h] = q * stride + elem_of_point(ax, i);
        off[h] = b0 + e;
      } else {
        const int i = e >> lt;
        valid = valid && v0;
        at[h] = (elem_of_point(ax, i) << lt) + q0;
        off[h] = b0 + (long)i * a.es;
      }
      if (!valid) off[h] = -1;
      x[h] = make_float2(valid ? in[off[h]] : 0.0f, (valid && two) ? in[a.fs + off[h]] : 0.0f);
    }
#pragma unroll
    for (int h = 0; h < UB; ++h) {
      if (off[h] < 0) continue;
      const float2 w = buf[at[h]];
      out[off[h]] = (x[h].x - w.x) + ea;
      if (two) out[a.fs + off[h]] = (x[h].y - w.y) + eb;
    }
  }
}

// ---------------------------------------------------------------- launch shapes
constexpr int kSmemMax = 226 * 1024;  // dynamic; a few static bytes beside it

int threads_for(long items) {  // whole warps, enough for a pass's butterflies
  long t = (items + 31) / 32 * 32;
  return (int)(t < 64 ? 64 : t > kThreads ? kThreads : t);
}

// Threads of a strided CTA (2^lt columns, nsig signals): the fewest rounds of
// butterflies over all passes, weighted by their radix; the smaller block
// where that does not tell.
int strided_threads(const SpecAxis& ax, int lt, int nsig) {
  int best = 64;
  long cost = -1;
  for (int t = 64; t <= kWide; t += 32) {
    const int W = t >> lt;
    if (W < 1) continue;
    long c = 0;
    for (int s = 0; s < ax.nst; ++s) {
      const int R = ax.radix[s], nb = ax.n / R;
      const int rounds = (W >= 2 * nb) ? (nsig + W / nb - 1) / (W / nb) : nsig * ((nb + W - 1) / W);
      c += (long)rounds * R;
    }
    if (cost < 0 || c < cost) {
      cost = c;
      best = t;
    }
  }
  return best;
}

// log2 of the columns per CTA: the widest of 16, 8, 4 and 2 whose tiles fit
// twice into an SM's shared memory (else once) and still give two CTAs per SM.
int strided_lt(const SpecAxis& ax, int nsig, long ncol, long outer, size_t* smem) {
  auto bytes = [&](int lt) { return ((size_t)nsig * (ax.len << lt) + 2 * ax.n) * sizeof(float2); };
  int best = 1;
  for (int lt = 4; lt >= 1; --lt) {
    if (bytes(lt) > (lt > 2 ? (size_t)kSmemMax / 2 : (size_t)kSmemMax)) continue;
    best = lt;
    if (((ncol + (1 << lt) - 1) >> lt) * outer >= 2 * 148) break;
  }
  *smem = bytes(best);
  return best;
}

}  // namespace

bool spec_factor(int n, int* radix, int* nst) {
  static const int R[] = {16, 15, 12, 10, 9, 8, 6, 5, 4, 3, 2};
  // fewest passes, then the smallest largest radix (depth-first over
  // non-increasing radices)
  std::vector<int> best, cur;
  struct Rec {
    static void go(int n, int from, std::vector<int>& cur, std::vector<int>& best) {
      if (n == 1) {
        if (best.empty() || cur.size() < best.size() || (cur.size() == best.size() && cur[0] < best[0])) best = cur;
        return;
      }
      if (!best.empty() && cur.size() >= best.size()) return;
      for (int i = from; i < 11; ++i)
        if (n % R[i] == 0) {
          cur.push_back(R[i]);
          go(n / R[i], i, cur, best);
          cur.pop_back();
        }
    }
  };
  Rec::go(n, 0, cur, best);
  if (best.empty() || best.size() > 8) return false;
  *nst = (int)best.size();
  for (size_t s = 0; s < best.size(); ++s) radix[s] = best[s];
  return true;
}

void spec_twiddles(int n, const int* radix, int nst, float2* tw) {
  int L = n;
  for (int s = 0; s < nst; ++s) {
    const int m = L / radix[s];
    for (int q = 1; q < radix[s]; ++q)
      for (int i = 0; i < m; ++i) {
        const double ang = -2.0 * M_PI * (double)((long)i * q % L) / L;
        tw[n - L + (q - 1) * m + i] = make_float2((float)cos(ang), (float)sin(ang));
      }
    L = m;
  }
  tw[n - 1] = make_float2(1.0f, 0.0f);
}

void spec_layout(const int* radix, int nst, int* len, int* st) {
  st[nst - 1] = 1;
  for (int s = nst - 2; s >= 0; --s) st[s] = (radix[s + 1] * st[s + 1]) | 1;
  *len = radix[0] * st[0];
}

namespace {
size_t x_bytes(int nd, int n, int len, int pg, bool flux) {
  const int nj = nd == 2 ? 2 : 3;
  const size_t sig = (size_t)(nd == 2 && flux ? 2 * nj : nj) * pg * len + 2 * n;
  return sig * sizeof(float2) + (nd == 3 && flux ? (size_t)5 * pg * n * sizeof(float) : 0);
}

template <int ND, bool INC, bool FLUX>
cudaError_t mrs_x(const SpecXArgs& a, const SpecAxis& ax, cudaStream_t s) {
  // rows per CTA: enough butterflies for 256 threads, a divisor of the rows
  // of a solve, at most half an SM's shared memory unless one row needs more
  const int nsig = (ND == 2) ? (FLUX ? 4 : 2) : 3;
  const int rmax = ax.radix[0];
  int pg = 1;
  while (2 * pg <= 64 && a.rps % (2 * pg) == 0 && (long)nsig * pg * (ax.n / rmax) < 256 &&
         x_bytes(ND, ax.n, ax.len, 2 * pg, FLUX) <= kSmemMax / 2 && a.rows / (2 * pg) >= 2 * 148)
    pg *= 2;
  const size_t sm = x_bytes(ND, ax.n, ax.len, pg, FLUX);
  cudaError_t e;
  if ((e = set_smem(k_mrs_x<ND, INC, FLUX>, kSmemMax)) != cudaSuccess) return e;
  return launch_dep(k_mrs_x<ND, INC, FLUX>, a.rows / pg, threads_for((long)nsig * pg * (ax.n / rmax)), sm, s, a, ax, pg);
}
}  // namespace

bool mrs_x_fits(int nd, int n) {
  int radix[16], nst, len, st[8];
  if (!spec_factor(n, radix, &nst)) return false;
  spec_layout(radix, nst, &len, st);
  return x_bytes(nd, n, len, 1, true) <= (size_t)kSmemMax;
}

cudaError_t launch_mrs_x(int nd, bool inc, bool flux, const SpecXArgs& a, const SpecAxis& ax, cudaStream_t s) {
  if (nd == 2) return inc ? (flux ? mrs_x<2, true, true>(a, ax, s) : mrs_x<2, true, false>(a, ax, s)) : mrs_x<2, false, true>(a, ax, s);
  return inc ? (flux ? mrs_x<3, true, true>(a, ax, s) : mrs_x<3, true, false>(a, ax, s)) : mrs_x<3, false, true>(a, ax, s);
}

#define PS_MRS_STRIDED(NAME, ARGS, KERNEL, NSIG, OUTER)                                        \
  cudaError_t NAME(const ARGS& a, const SpecAxis& ax, cudaStream_t s) {                        \
    size_t sm = 0;                                                                             \
    const int lt = strided_lt(ax, NSIG, a.ncol, OUTER, &sm);                                   \
    const int threads = strided_threads(ax, lt, NSIG);                                         \
    const long ctas = (long)((a.ncol + (1 << lt) - 1) >> lt) * (OUTER);                        \
    if (ctas > INT_MAX) return cudaErrorInvalidConfiguration;                                  \
    const int grid = (int)ctas;                                                                \
    cudaError_t e;                                                                             \
    if (threads > kThreads) {                                                                  \
      if ((e = set_smem(KERNEL<kWide>, kSmemMax)) != cudaSuccess) return e;                    \
      return launch_dep(KERNEL<kWide>, grid, threads, sm, s, a, ax, lt);                       \
    }                                                                                          \
    if ((e = set_smem(KERNEL<kThreads>, kSmemMax)) != cudaSuccess) return e;                   \
    return launch_dep(KERNEL<kThreads>, grid, threads, sm, s, a, ax, lt);                      \
  }
PS_MRS_STRIDED(launch_mrs_f, SpecFArgs, k_mrs_f, 2, a.planes)
PS_MRS_STRIDED(launch_mrs_c, SpecCArgs, k_mrs_c, 2, (long)a.nouter * a.nsolve)
PS_MRS_STRIDED(launch_mrs_i, SpecIArgs, k_mrs_i, 1, a.planes)

namespace {
// Registers of the filter pass: 128 a thread while all CTAs run at once that way,
// else 64 (with a few spills), where more of them fit an SM beside one another.
// 128 against 64: 480^2 46.0 / 49.3 us, 96 x 90 x 32 35.7 / 39.2; 540 x 960 84.5 /
// 58.0, 90 x 96 x 100 177 / 133, 250^2 x 32 240 / 178, 3840 x 2160 795 / 736.
template <bool ROWS>
cudaError_t mrs_filter(const MrFilterArgs& a, const SpecAxis& ax, dim3 grid, int threads, size_t sm, int lt,
                       cudaStream_t s) {
  cudaError_t e;
  auto per_sm = [&](int regs) { return std::min(65536 / (regs * threads), (int)((227 * 1024) / (sm + 1024))); };
  if (per_sm(64) > per_sm(128) && (long)grid.x * grid.y * grid.z > 152L * per_sm(128)) {
    if ((e = set_smem(k_mrs_filter<ROWS, 2>, kSmemMax)) != cudaSuccess) return e;
    return launch_dep(k_mrs_filter<ROWS, 2>, grid, threads, sm, s, a, ax, lt);
  }
  if ((e = set_smem(k_mrs_filter<ROWS, 1>, kSmemMax)) != cudaSuccess) return e;
  return launch_dep(k_mrs_filter<ROWS, 1>, grid, threads, sm, s, a, ax, lt);
}
}  // namespace

cudaError_t launch_mrs_filter(const MrFilterArgs& a, const SpecAxis& ax, int nsolve, cudaStream_t s) {
  const int rmax = ax.radix[0], pairs = (a.nf + 1) / 2;
  auto tiles = [&](int l) { return (a.npen + (1L << l) - 1) >> l; };
  auto bytes = [&](int l) { return ((size_t)(ax.len << l) + 2 * ax.n) * sizeof(float2); };
  // one more doubling of the pencils per CTA, while that leaves two CTAs per SM
  auto wider = [&](int l) { return tiles(l) > 1 && tiles(l + 1) * pairs * nsolve >= 2 * 152; };
  const bool rows = a.es == 1;
  int lt = 0;
  size_t sm;
  if (rows) {
    while (lt < 6 && ((long)(ax.n / rmax) << lt) < 256 && bytes(lt + 1) <= kSmemMax / 3 && wider(lt)) ++lt;
  } else {  // short axes: tiles of up to 1024 points
    lt = strided_lt(ax, 1, a.npen, (long)pairs * nsolve, &sm);
    while (lt >= 4 && lt < 8 && (ax.n << (lt + 1)) <= 1024 && wider(lt)) ++lt;
  }
  sm = bytes(lt);
  const dim3 grid((unsigned)tiles(lt), nsolve, pairs);
  const int threads = threads_for((long)(ax.n / rmax) << lt);
  return rows ? mrs_filter<true>(a, ax, grid, threads, sm, lt, s) : mrs_filter<false>(a, ax, grid, threads, sm, lt, s);
}

}  // namespace ps

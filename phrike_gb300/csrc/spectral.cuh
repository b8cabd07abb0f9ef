// Fixed-step and CFL stepping of 2D/3D Euler and MHD on power-of-two Fourier
// grids with the flux spectra kept truncated between the passes.
//
// The separable operators (euler_passes.cuh) are applied to every axis by one
// forward transform only; the inverse transforms act on the contracted
// right-hand side alone.  Per RK stage:
//   k_spec_x (x rows)      : U_s = U^n + increment (inverse x transform of its
//                            spectra), clamp, fluxes, forward x transforms,
//                            G_d = D_x F^x, P_x F^y, P_x F^z
//   k_spec_f (y, 3D only)  : forward y, A = P_y G_x + D_y G_y, B = P_y G_z
//   k_spec_c (last axis)   : forward, k = -(P A + D B), RK accumulator in
//                            spectral space, stage increment, inverse
//   k_spec_i (y, 3D only)  : inverse y of the increment
// The dealias mask drops every mode above N/3 before a pass stores its
// output, so a transformed axis holds M = 2 (N/3) + 1 of its N modes: the
// intermediate arrays carry 2/3 of the real-space words per transformed axis
// and the later transforms run on 2/3 of the pencils.  Against the passes
// that return to real space after each axis a 3D Euler stage moves 49 words
// per cell instead of 75 and runs 22 complex pencil transforms per cell
// instead of 37; a 3D MHD stage moves 77 words instead of 230 (and needs no
// projection per stage, see steps_spec).  Measured per step against those
// passes, with what the kernels below gained since: Taylor-Green 256^3 (mask
// filter) 4.95 -> 3.23 ms, KHI 512^2 x 16 1.06 -> 0.72 ms, Orszag-Tang 512^2
// 0.456 -> 0.180 ms, 3D MHD 128^3 2.29 -> 0.98 ms.  Traffic bounds the y and z
// passes (Taylor-Green 256^3: y forward 173 us at 5.4 TB/s, last 128 us, y
// inverse 66 us) and instruction issue the x pass (349 us for 1.24 GB, 12
// transforms per row at 12 warps per SM).
//
// Two real fields travel as one complex field: every operator maps real
// fields to real fields, so it acts on f + i g as on f and g, and no pass but
// the x inverse ever looks at the halves.  A "wide" row holds the columns of
// all component pairs side by side, [pair][mode m]; m counts the kept modes,
// 0..KM then -KM..-1.  The fifth field of 3D Euler (the energy) stands alone
// and stores its non-negative modes only.  The y and z passes see plain
// columns and do not depend on the equations.
#pragma once
#include "euler_passes.cuh"
#include "mhd_passes.cuh"
#include "tma.cuh"

namespace ps {

// Kept modes of a masked axis and the shape of a wide row.
__host__ __device__ constexpr int spec_km(int n) { return n / 3; }
__host__ __device__ constexpr int spec_modes(int n) { return 2 * (n / 3) + 1; }
// columns of a wide row: full pairs, then half spectra of a single last field
__host__ __device__ constexpr int spec_cols(int nx, int nc) {
  return (nc / 2) * spec_modes(nx) + (nc % 2) * (spec_km(nx) + 1);
}
// row pitch in complex elements (64-byte rows)
__host__ __device__ constexpr int spec_pitch(int nx, int nc) { return (spec_cols(nx, nc) + 7) / 8 * 8; }

struct SpecXArgs {
  const float* U;     // U^n [nsolve][NC][cells]
  float* Uw;          // nullable: the state after the x filter (no increment) or after the increment is written here
  const float* Bp;    // MHD, nullable: [nsolve][nproj][cells], the projected B of U^n
  int nproj;          // fields of B the projection covers (2 in 2D, 3 in 3D)
  const float2* D;    // increment spectra, wide rows (with an increment)
  float2* G;          // flux spectra, ND wide arrays
  long gs;            // complex elements between the arrays of G
  int pitch;          // complex elements per wide row
  long fs, ssU;       // elements per field, per solve
  int rows, rps;      // rows of all solves, of one solve
  AxisOps ax;
  float gamma;
  float rho_min, p_min;
  float* speed;       // nullable: per-solve max wave speed of the state the fluxes are taken of
  const float* eref;  // Euler: E_ref per solve
  const int* active;
  int px;             // apply the complementary x filter to the loaded state and write it to Uw
  int shift_in;       // U holds E (subtract E_ref on load)
  int shift_out;      // Uw takes E (add E_ref on store)
};

template <int N, int T>
struct SpecXSmem {
  AxisSmem<N> ax;
  float2 buf[Pencil<N, T, false>::BUF];
  float red[32];
};

// Column of mode k (0..N-1) inside one pair's M columns, or -1 if masked.
template <int N>
__device__ __forceinline__ int spec_col(int k) {
  constexpr int KM = spec_km(N);
  if (k <= KM) return k;
  if (k >= N - KM) return k - (N - 2 * KM - 1);
  return -1;
}
// Whether register r of a pencil thread can hold a kept mode (compile time;
// N <= 256: k = t + A (r / A) + B (r % A), t in [0, A)).  Transforms whose
// masked outputs are never read lose the butterflies that produce them.
template <int N>
constexpr bool spec_keeps(int r) {
  if (N > 256) return true;
  const int lo = Shape<N>::A * (r / Shape<N>::A) + Shape<N>::B * (r % Shape<N>::A);
  const int hi = lo + Shape<N>::A - 1;
  return lo <= spec_km(N) || hi >= N - spec_km(N);
}

template <int DIR, int C>
__device__ __forceinline__ float mhd3_flux(float rho, float ux, float uy, float uz, float ps, float eps, float ub,
                                           float Bx, float By, float Bz) {
  const float un = (DIR == 0) ? ux : (DIR == 1) ? uy : uz;
  const float Bn = (DIR == 0) ? Bx : (DIR == 1) ? By : Bz;
  const float mn = rho * un;
  if constexpr (C == 0) return mn;
  if constexpr (C == 1) return mn * ux + ((DIR == 0) ? ps : 0.0f) - Bn * Bx;
  if constexpr (C == 2) return mn * uy + ((DIR == 1) ? ps : 0.0f) - Bn * By;
  if constexpr (C == 3) return mn * uz + ((DIR == 2) ? ps : 0.0f) - Bn * Bz;
  if constexpr (C == 4) return eps * un - Bn * ub;
  if constexpr (C == 5) return (DIR == 0) ? 0.0f : un * Bx - ux * Bn;
  if constexpr (C == 6) return (DIR == 1) ? 0.0f : un * By - uy * Bn;
  return (DIR == 2) ? 0.0f : un * Bz - uz * Bn;  // C == 7
}

// Conservative to primitive at one point (rho, u, p' for Euler; B and E stay
// for MHD); returns the wave speed of the point, or 0 if not asked for.  The
// Euler products that meet a sum here and in the fluxes are rounded as
// written: left to the compiler, the two kernels of the x rows contracted them
// differently (wave speeds at 8 points per row), and a solve must give the
// same bits alone and in a batch.
template <int ND, int PHYS, int NC>
__device__ __forceinline__ float spec_primitive(float (&u)[NC], float gamma, float g1, float pref, bool speed) {
  constexpr int NV = (PHYS == 1) ? 3 : ND;
  const float rho = u[0];
  const float rinv = 1.0f / rho;
  float kin = 0.0f;
  float vel[NV];
#pragma unroll
  for (int d = 0; d < NV; ++d) {
    vel[d] = u[1 + d] * rinv;
    kin = fmaf(vel[d], vel[d], kin);
    u[1 + d] = vel[d];
  }
  if constexpr (PHYS == 0) {
    const float pr = __fmul_rn(g1, fmaf(-0.5f * rho, kin, u[NC - 1]));
    u[NC - 1] = pr;
    if (!speed) return 0.0f;
    const float cs = sqrtf(gamma * __fadd_rn(pr, pref) * rinv);
    float um = fabsf(vel[0]);
    if (ND == 3) um = fmaxf(um, fmaxf(fabsf(vel[1]), fabsf(vel[NV - 1])));
    return um + cs;  // 2D keeps |u_x| + a only (equations.py:137-147)
  } else {  // equations.py:874-887, 1040-1061
    if (!speed) return 0.0f;
    const float b2 = u[5] * u[5] + u[6] * u[6] + u[7] * u[7];
    const float pr = g1 * (u[4] - 0.5f * rho * kin - 0.5f * b2);
    float um = fmaxf(fabsf(vel[0]), fabsf(vel[1]));
    if (ND == 3) um = fmaxf(um, fabsf(vel[2]));
    return um + sqrtf(fmaxf(gamma * pr / rho + b2 / rho, 0.0f));
  }
}

// total pressure and u . B of MHD primitives (rho, u, E, B)
__device__ __forceinline__ void mhd_derived(const float (&u)[8], float g1, float& ps, float& ub) {
  const float b2 = u[5] * u[5] + u[6] * u[6] + u[7] * u[7];
  const float v2 = u[1] * u[1] + u[2] * u[2] + u[3] * u[3];
  ps = g1 * (u[4] - 0.5f * u[0] * v2 - 0.5f * b2) + 0.5f * b2;
  ub = u[1] * u[5] + u[2] * u[6] + u[3] * u[7];
}

// Largest speed of a tile's T rows into their solves' slots (all threads)
__device__ __forceinline__ void spec_speed(const SpecXArgs& a, float smax, bool valid, int sol, int tile, int T,
                                           float* red) {
  const int s0 = (tile * T) / a.rps;
  const int s1 = (min(tile * T + T, a.rows) - 1) / a.rps;
  if (s0 == s1) {
    const float m = block_max(smax, red);
    if (threadIdx.x == 0) atomic_max_nonneg(a.speed + s0, m);
  } else if (valid) {  // rows of several small solves in one CTA
    atomic_max_nonneg(a.speed + sol, smax);
  }
}

// Flux jobs first, first + step, .. of a row whose primitives are q(c, n2):
// fluxes of a component pair along one direction, forward transform, D_x or
// P_x, store.  opaque() keeps the compiler from carrying flux terms over the
// jobs.  DERIVED (MHD): q(4) is E plus the total pressure, q(8) the total
// pressure and q(9) u . B, so that the jobs do not each take them again.
template <int N, int T, int ND, int PHYS, bool DERIVED, typename PF, typename Q, typename O>
__device__ __forceinline__ void spec_fluxes(const SpecXArgs& a, const PF& pf, const AxisSmem<N>& ax,
                                            Q&& q, O&& opaque, float er, int row, bool valid, int first, int step) {
  constexpr int B = Shape<N>::B;
  constexpr int NC = (PHYS == 1) ? 8 : ND + 2;
  constexpr int NP = NC / 2;
  constexpr bool ODD = (NC % 2) != 0;
  constexpr int NJ = NP + (ODD ? 1 : 0);
  constexpr int KM = spec_km(N), M = spec_modes(N);
  const float g1 = a.gamma - 1.0f;
  auto put = [&](int j, auto&& f) {
    sfor<0, NJ>([&](auto jc) {
      if (j == decltype(jc)::value) f(jc);
    });
  };
  const float href = __fmul_rn(a.gamma, er);
  const float ig1 = 1.0f / g1;
  // Euler flux pair j = (F_2j, F_2j+1) along the (runtime) direction dir.
  // The direction enters by selects, so one body per pair serves the ND
  // directions (a third of the code: TGV 256^3 x pass 325 -> 321 us, KHI
  // 512^2 x 16 92 -> 89; the longer MHD bodies ran slower that way, 131 ->
  // 139 us at 128^3, and take the direction at compile time).
  auto flux_pair = [&](auto jc, int dir, int n2) -> float2 {
    constexpr int c = 2 * decltype(jc)::value;
    const float un = (dir == 0) ? q(1, n2) : (ND == 2 || dir == 1) ? q(2, n2) : q((ND == 3) ? 3 : 2, n2);
    const float mn = __fmul_rn(q(0, n2), un);
    auto comp = [&](auto cc) -> float {
      constexpr int C = decltype(cc)::value;
      const float pr = q(NC - 1, n2);
      if constexpr (C == 0) return mn;
      if constexpr (C == NC - 1) {
        float kin = 0.0f;
#pragma unroll
        for (int d = 0; d < ND; ++d) kin = fmaf(q(1 + d, n2), q(1 + d, n2), kin);
        const float Ep = fmaf(pr, ig1, __fmul_rn(0.5f * q(0, n2), kin));      // E' = E - E_ref
        return __fmul_rn(__fadd_rn(__fadd_rn(Ep, pr), href), un);  // (E + p) u_dir
      }
      return fmaf(mn, q(C, n2), (C - 1 == dir) ? pr : 0.0f);
    };
    float2 f = make_float2(comp(std::integral_constant<int, c>{}), 0.0f);
    if constexpr (c + 1 < NC) f.y = comp(std::integral_constant<int, c + 1>{});
    return f;
  };
#pragma unroll 1
  for (int job = first; job < ND * NJ; job += step) {
    opaque();
    const int dir = job / NJ, j = job % NJ;
    float2 v[B];
    if constexpr (PHYS == 1) {
      sfor<0, ND * NJ>([&](auto jobc) {
        constexpr int J = decltype(jobc)::value;
        constexpr int DIR = J / NJ, c = 2 * (J % NJ);
        if (job == J) {
#pragma unroll
          for (int n2 = 0; n2 < B; ++n2) {
            float ps, ub, eps;
            if constexpr (DERIVED) {
              eps = q(4, n2);
              ps = q(8, n2);
              ub = q(9, n2);
            } else {
              float u[8];
#pragma unroll
              for (int i = 0; i < 8; ++i) u[i] = q(i, n2);
              mhd_derived(u, g1, ps, ub);
              eps = u[4] + ps;
            }
            auto f = [&](auto cc) {
              return mhd3_flux<DIR, decltype(cc)::value>(q(0, n2), q(1, n2), q(2, n2), q(3, n2), ps, eps, ub, q(5, n2),
                                                         q(6, n2), q(7, n2));
            };
            v[n2] = make_float2(f(std::integral_constant<int, c>{}), f(std::integral_constant<int, c + 1>{}));
          }
        }
      });
    } else {
      put(j, [&](auto jc) {
#pragma unroll
        for (int n2 = 0; n2 < B; ++n2) v[n2] = flux_pair(jc, dir, n2);
      });
    }
    const bool single = ODD && j == NP;
    pf.fwd(v);
    float2* g = a.G + dir * a.gs + (long)row * a.pitch + j * M;
    sfor<0, B>([&](auto rc) {
      constexpr int r = decltype(rc)::value;
      if constexpr (spec_keeps<N>(r)) {
        const int k = pf.kidx(r);
        const int m = spec_col<N>(k);
        float2 w;
        if (dir == 0) {
          const float dd = ax.d[k];
          w = make_float2(-v[r].y * dd, v[r].x * dd);
        } else {
          const float s = ax.P[k];
          w = make_float2(v[r].x * s, v[r].y * s);
        }
        if (valid && m >= 0 && !(ODD && single && m > KM)) g[m] = w;
      }
    });
  }
}

// x rows.  INC: the state is U^n plus the increment of a.D; FLUX: fluxes of
// the state are transformed and stored.  The thread's B points of every
// component stay in registers (q[c][n2]); a switch over the job index keeps
// one transform body for all jobs.  PHYS 0 Euler, 1 MHD (8 components).
template <int N, int T, int ND, int PHYS, bool INC, bool FLUX>
__global__ void __launch_bounds__(Shape<N>::A * T) k_spec_x(SpecXArgs a) {
  constexpr int NC = (PHYS == 1) ? 8 : ND + 2;
  constexpr int NP = NC / 2;            // packed pairs
  constexpr bool ODD = (NC % 2) != 0;   // a single last field
  constexpr int NJ = NP + (ODD ? 1 : 0);
  constexpr int A = Shape<N>::A, B = Shape<N>::B;
  constexpr int KM = spec_km(N), M = spec_modes(N);
  using PF = Pencil<N, T, false>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  auto& S = *reinterpret_cast<SpecXSmem<N, T>*>(smem_raw);

  load_axis<N>(S.ax, a.ax);
  dep_wait();
  const int t = threadIdx.x % A;
  const int p = threadIdx.x / A;
  const int row = blockIdx.x * T + p;
  const int sol = (row < a.rows ? row : a.rows - 1) / a.rps;
  const bool live = a.active == nullptr || a.active[sol] != 0;
  const bool valid = row < a.rows && live;
  {  // a CTA whose rows all belong to inactive solves has nothing to do
    const int r0 = blockIdx.x * T, r1 = min(r0 + T, a.rows) - 1;
    bool any = a.active == nullptr;
    for (int s2 = r0 / a.rps; !any && s2 <= r1 / a.rps; ++s2) any = a.active[s2] != 0;
    if (!any) return;
  }
  PF pf{p, t, S.buf, S.ax.twf, S.ax.twi};
  const long rbase = (long)sol * a.ssU + (long)(row % a.rps) * N + t;
  const float er = (PHYS == 0) ? a.eref[sol] : 0.0f;
  const float eshift = a.shift_in ? er : 0.0f;
  const float g1 = a.gamma - 1.0f;
  const float pref = __fmul_rn(g1, er);
  constexpr int CE = (PHYS == 1) ? 4 : NC - 1;  // energy component
  float q[NC][B];
#pragma unroll
  for (int c = 0; c < NC; ++c) {
#pragma unroll
    for (int n2 = 0; n2 < B; ++n2) {
      float v = (c == 0) ? 1.0f : 0.0f;
      if (valid) v = a.U[c * a.fs + rbase + A * n2];  // may alias a.Uw: plain load
      if (PHYS == 0 && c == CE && valid) v -= eshift;
      q[c][n2] = v;
    }
  }
  __syncthreads();

  // q[c] (and q[c + 1]) <- op on the pair of job j
  auto put = [&](int j, auto&& f) {
    sfor<0, NJ>([&](auto jc) {
      constexpr int J = decltype(jc)::value;
      if (j == J) f(jc);
    });
  };

  if constexpr (INC) {
    const float2* Drow = a.D + (long)row * a.pitch;
#pragma unroll 1
    for (int j = 0; j < NJ; ++j) {
      float2 v[B];
      const bool single = ODD && j == NP;
      const float2* d = Drow + j * M;
      sfor<0, B>([&](auto rc) {
        constexpr int r = decltype(rc)::value;
        v[r] = make_float2(0.0f, 0.0f);
        if constexpr (spec_keeps<N>(r)) {
          const int k = pf.kidx(r);
          int m = spec_col<N>(k);
          if (ODD && single && m > KM) m = N - k;  // half spectra: X(-k) = conj X(k)
          if (valid && m >= 0) v[r] = d[m];
          if (ODD && single && k > KM) v[r].y = -v[r].y;
        }
      });
      pf.inv(v);
      put(j, [&](auto jc) {
        constexpr int c = 2 * decltype(jc)::value;
        constexpr bool two = c + 1 < NC;
#pragma unroll
        for (int n2 = 0; n2 < B; ++n2) {
          q[c][n2] += v[n2].x;
          if constexpr (two) q[c + 1][n2] += v[n2].y;
        }
      });
    }
    if constexpr (PHYS == 1) {
#pragma unroll
      for (int n2 = 0; n2 < B; ++n2) {
        float u[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) u[c] = q[c][n2];
        clamp_mhd(u, a.gamma, a.rho_min, a.p_min);
        // the stage projection: the increment of B is solenoidal mode by mode
        // (the induction flux u_i B_j - u_j B_i is antisymmetric), so it only
        // replaces U^n's B by its projection; E keeps the thermal pressure
        if (a.Bp != nullptr && valid) {
#pragma unroll
          for (int c = 5; c < 8; ++c) {
            if (c - 5 >= a.nproj) break;
            const long o = (long)(row % a.rps) * N + t + A * n2;  // within a field
            const float b = u[c] + (a.Bp[((long)sol * a.nproj + c - 5) * a.fs + o] - a.U[c * a.fs + rbase + A * n2]);
            u[4] += 0.5f * (b * b - u[c] * u[c]);
            u[c] = b;
          }
        }
#pragma unroll
        for (int c = 0; c < 8; ++c) q[c][n2] = u[c];
      }
    } else if constexpr (ND == 2) {
      const float pmin_shift = a.p_min - pref;
#pragma unroll
      for (int n2 = 0; n2 < B; ++n2) {
        float u[NC];
#pragma unroll
        for (int c = 0; c < NC; ++c) u[c] = q[c][n2];
        clamp_state<ND>(u, a.gamma, a.rho_min, pmin_shift);
#pragma unroll
        for (int c = 0; c < NC; ++c) q[c][n2] = u[c];
      }
    }
    if (a.Uw != nullptr && valid) {
      const float so = (PHYS == 0 && a.shift_out) ? er : 0.0f;
#pragma unroll
      for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int n2 = 0; n2 < B; ++n2)
          a.Uw[c * a.fs + rbase + A * n2] = (PHYS == 0 && c == CE) ? q[c][n2] + so : q[c][n2];
    }
  } else if (a.px) {  // fused x factor of the end-of-step filter (complementary form)
#pragma unroll 1
    for (int j = 0; j < NJ; ++j) {
      float2 v[B];
      put(j, [&](auto jc) {
        constexpr int c = 2 * decltype(jc)::value;
        constexpr int c1 = (c + 1 < NC) ? c + 1 : c;
#pragma unroll
        for (int n2 = 0; n2 < B; ++n2) v[n2] = make_float2(q[c][n2], (c + 1 < NC) ? q[c1][n2] : 0.0f);
      });
      pf.fwd(v);
#pragma unroll
      for (int r = 0; r < B; ++r) {
        const float s = (1.0f / N) - S.ax.P[pf.kidx(r)];
        v[r].x *= s;
        v[r].y *= s;
      }
      pf.inv(v);
      put(j, [&](auto jc) {
        constexpr int c = 2 * decltype(jc)::value;
        constexpr int c1 = (c + 1 < NC) ? c + 1 : c;
#pragma unroll
        for (int n2 = 0; n2 < B; ++n2) {
          q[c][n2] -= v[n2].x;
          if (valid) a.Uw[c * a.fs + rbase + A * n2] = q[c][n2];
          if constexpr (c + 1 < NC) {
            q[c1][n2] -= v[n2].y;
            if (valid) a.Uw[c1 * a.fs + rbase + A * n2] = q[c1][n2];
          }
        }
      });
    }
  }
  if constexpr (FLUX) {
    float smax = 0.0f;
#pragma unroll
    for (int n2 = 0; n2 < B; ++n2) {
      float u[NC];
#pragma unroll
      for (int c = 0; c < NC; ++c) u[c] = q[c][n2];
      smax = fmaxf(smax, spec_primitive<ND, PHYS>(u, a.gamma, g1, pref, a.speed != nullptr && valid));
#pragma unroll
      for (int c = 0; c < NC; ++c) q[c][n2] = u[c];
    }
    if (a.speed != nullptr) spec_speed(a, smax, valid, sol, blockIdx.x, T, S.red);
    // the state's registers are opaque per job: without this the compiler
    // keeps flux terms shared by several jobs live across the loop (16
    // registers each) and spills
    auto opaque = [&]() {
#pragma unroll
      for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int n2 = 0; n2 < B; ++n2) asm volatile("" : "+f"(q[c][n2]));
    };
    spec_fluxes<N, T, ND, PHYS, false>(a, pf, S.ax, [&](int c, int n2) { return q[c][n2]; }, opaque, er, row, valid, 0,
                                       1);
  }
}

// x rows of MHD and of Euler grids with few pencils: a warp per pencil group
// and job group.  k_spec_x takes a row through all its transforms in one warp.
// That leaves most of the GPU idle when the rows are few (128 rows of 128
// points are 32 warps for 152 SMs, each with a chain of 6 transforms), and the
// 128 registers of an MHD state leave two CTAs per SM.  Here NG job groups
// share the rows of a CTA: each takes its component pairs through the inverse
// transform, the state meets in shared memory, the points are dealt over all
// threads for the clamp and the primitives, and each group takes its share of
// the flux transforms.  The arithmetic per value is that of k_spec_x.
template <int N, int T, int NC, int NG>
struct SpecXsSmem {
  AxisSmem<N> ax;
  float2 buf[NG][Pencil<N, T, false>::BUF];
  float q[(NC == 8) ? 10 : NC][T * N];  // [component (and MHD's derived values)][n2][thread of the group]
  float red[32];
};

template <int N, int ND, int PHYS, int NG, bool INC, bool FLUX>
__global__ void __launch_bounds__(32 * NG, (PHYS == 1) ? 4 : 0) k_spec_xs(SpecXArgs a) {
  constexpr int NC = (PHYS == 1) ? 8 : ND + 2;
  constexpr int NP = NC / 2;
  constexpr bool ODD = (NC % 2) != 0;
  constexpr int NJ = NP + (ODD ? 1 : 0);
  constexpr int A = Shape<N>::A, B = Shape<N>::B, T = 32 / A;
  constexpr int KM = spec_km(N), M = spec_modes(N);
  using PF = Pencil<N, T, false>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  auto& S = *reinterpret_cast<SpecXsSmem<N, T, NC, NG>*>(smem_raw);
  load_axis<N>(S.ax, a.ax);
  dep_wait();
  const int grp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int t = lane % A, p = lane / A;
  PF pf{p, t, S.buf[grp], S.ax.twf, S.ax.twi};
  auto tile_rows = [&](int tile) {
    const int row = tile * T + p;
    const int sol = (row < a.rows ? row : a.rows - 1) / a.rps;
    const bool valid = row < a.rows && (a.active == nullptr || a.active[sol] != 0);
    if (a.active != nullptr) {
      bool any = false;
      for (int s2 = tile * T / a.rps; !any && s2 <= (min(tile * T + T, a.rows) - 1) / a.rps; ++s2)
        any = a.active[s2] != 0;
      if (!any) return;
    }
    const long rbase = (long)sol * a.ssU + (long)(row % a.rps) * N + t;
    const float er = (PHYS == 0) ? a.eref[sol] : 0.0f;
    const float eshift = a.shift_in ? er : 0.0f;
    const float g1 = a.gamma - 1.0f;
    const float pref = __fmul_rn(g1, er);
    constexpr int CE = (PHYS == 1) ? 4 : NC - 1;
    auto slot = [&](int c, int n2) -> float& { return S.q[c][n2 * 32 + lane]; };
    // this thread's points in the middle part are n2 = grp + NG i; the stage
    // projection's change of U^n there is loaded ahead of the transforms
    constexpr int NPT = (B + NG - 1) / NG;
    [[maybe_unused]] float dB[NPT][3];
    if constexpr (INC && PHYS == 1) {
#pragma unroll
      for (int i = 0; i < NPT; ++i)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const int n2 = grp + NG * i;
          const long o = (long)(row % a.rps) * N + t + A * n2;  // within a field
          dB[i][c] = (a.Bp != nullptr && valid && n2 < B && c < a.nproj)
                         ? a.Bp[((long)sol * a.nproj + c) * a.fs + o] - a.U[(5 + c) * a.fs + rbase + A * n2]
                         : 0.0f;
        }
    }
    __syncthreads();  // the tables; the state's last readers

    // the group's component pairs: U^n (plus the increment, or filtered along x)
#pragma unroll 1
    for (int j = grp; j < NJ; j += NG) {
      const bool single = ODD && j == NP;
      const int c0 = 2 * j, c1 = single ? c0 : c0 + 1;
      float2 u[B], v[B];
#pragma unroll
      for (int n2 = 0; n2 < B; ++n2) {
        u[n2].x = valid ? a.U[c0 * a.fs + rbase + A * n2] : (c0 == 0 ? 1.0f : 0.0f);
        u[n2].y = (valid && !single) ? a.U[c1 * a.fs + rbase + A * n2] : 0.0f;
        if (PHYS == 0 && valid) {
          if (c0 == CE) u[n2].x -= eshift;
          else if (c1 == CE) u[n2].y -= eshift;
        }
      }
      if constexpr (INC) {
        const float2* d = a.D + (long)row * a.pitch + j * M;
        sfor<0, B>([&](auto rc) {
          constexpr int r = decltype(rc)::value;
          v[r] = make_float2(0.0f, 0.0f);
          if constexpr (spec_keeps<N>(r)) {
            const int k = pf.kidx(r);
            int m = spec_col<N>(k);
            if (ODD && single && m > KM) m = N - k;  // half spectra: X(-k) = conj X(k)
            if (valid && m >= 0) v[r] = d[m];
            if (ODD && single && k > KM) v[r].y = -v[r].y;
          }
        });
        pf.inv(v);
#pragma unroll
        for (int n2 = 0; n2 < B; ++n2) {
          u[n2].x += v[n2].x;
          u[n2].y += v[n2].y;
        }
      } else if (a.px) {
#pragma unroll
        for (int n2 = 0; n2 < B; ++n2) v[n2] = u[n2];
        pf.fwd(v);
#pragma unroll
        for (int r = 0; r < B; ++r) {
          const float s = (1.0f / N) - S.ax.P[pf.kidx(r)];
          v[r].x *= s;
          v[r].y *= s;
        }
        pf.inv(v);
#pragma unroll
        for (int n2 = 0; n2 < B; ++n2) {
          u[n2].x -= v[n2].x;
          u[n2].y -= v[n2].y;
          if (valid) {
            a.Uw[c0 * a.fs + rbase + A * n2] = u[n2].x;
            if (!single) a.Uw[c1 * a.fs + rbase + A * n2] = u[n2].y;
          }
        }
      }
#pragma unroll
      for (int n2 = 0; n2 < B; ++n2) {
        slot(c0, n2) = u[n2].x;
        if (!single) slot(c1, n2) = u[n2].y;
      }
    }
    __syncthreads();

    // points n2 = grp, grp + NG, ..: clamp, new state, primitives
    float smax = 0.0f;
#pragma unroll
    for (int i = 0; i < NPT; ++i) {
      const int n2 = grp + NG * i;
      if (n2 >= B) break;
      float u[NC];
#pragma unroll
      for (int c = 0; c < NC; ++c) u[c] = slot(c, n2);
      if constexpr (INC) {
        if constexpr (PHYS == 1) {
          clamp_mhd(u, a.gamma, a.rho_min, a.p_min);
          if (a.Bp != nullptr && valid) {
#pragma unroll
            for (int c = 5; c < 8; ++c) {
              if (c - 5 >= a.nproj) break;
              const float b = u[c] + dB[i][c - 5];
              u[4] += 0.5f * (b * b - u[c] * u[c]);
              u[c] = b;
            }
          }
        } else if constexpr (ND == 2) {
          const float pmin_shift = a.p_min - pref;
          clamp_state<ND>(u, a.gamma, a.rho_min, pmin_shift);
        }
        if (a.Uw != nullptr && valid) {
          const float so = (PHYS == 0 && a.shift_out) ? er : 0.0f;
#pragma unroll
          for (int c = 0; c < NC; ++c)
            a.Uw[c * a.fs + rbase + A * n2] = (PHYS == 0 && c == CE) ? u[c] + so : u[c];
        }
      }
      if constexpr (FLUX) {
        smax = fmaxf(smax, spec_primitive<ND, PHYS>(u, a.gamma, g1, pref, a.speed != nullptr && valid));
        if constexpr (PHYS == 1) {
          float ps, ub;
          mhd_derived(u, g1, ps, ub);
          u[4] += ps;
          slot(8, n2) = ps;
          slot(9, n2) = ub;
        }
#pragma unroll
        for (int c = 0; c < NC; ++c) slot(c, n2) = u[c];
      }
    }
    if constexpr (FLUX) {
      if (a.speed != nullptr) spec_speed(a, smax, valid, sol, tile, T, S.red);
      __syncthreads();
      if constexpr (PHYS == 1) {
        // points come from shared memory per job: the whole state in registers
        // (128 of them) leaves half the warps in flight.  Orszag-Tang 512^2 step
        // 200 -> 183 us; the 16 to 80 registers of the Euler states stay
        spec_fluxes<N, T, ND, PHYS, true>(a, pf, S.ax, slot, [] { asm volatile("" ::: "memory"); }, er, row, valid, grp, NG);
      } else {
        float q[NC][B];
#pragma unroll
        for (int c = 0; c < NC; ++c)
#pragma unroll
          for (int n2 = 0; n2 < B; ++n2) q[c][n2] = slot(c, n2);
        auto opaque = [&] {  // as in k_spec_x
#pragma unroll
          for (int c = 0; c < NC; ++c)
#pragma unroll
            for (int n2 = 0; n2 < B; ++n2) asm volatile("" : "+f"(q[c][n2]));
        };
        spec_fluxes<N, T, ND, PHYS, false>(a, pf, S.ax, [&](int c, int n2) { return q[c][n2]; }, opaque, er, row, valid, grp, NG);
      }
    }
  };
  if constexpr (PHYS == 1) {
    // a CTA walks over its tiles, the tables loaded once; the loop costs the
    // Euler kernels 10 to 30 registers (Taylor-Green 64^3 92.8 -> 99 us)
#pragma unroll 1
    for (int tile = blockIdx.x; tile < (a.rows + T - 1) / T; tile += gridDim.x) tile_rows(tile);
  } else {
    tile_rows(blockIdx.x);
  }
}

// ---------------------------------------------------------------------------
// Strided passes over wide columns: T adjacent columns per tile, A threads per
// column.  A CTA walks over its share of the tiles; cp.async copies (16 bytes,
// two columns) bring the next tile's points into shared memory while the
// present one is transformed, so the transforms do not wait for memory.  A
// tile row is T * 8 bytes; rows are 64-byte aligned (spec_pitch).
// ---------------------------------------------------------------------------
__device__ __forceinline__ void cp16(void* dst, const void* src, bool take) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_addr(dst)), "l"(src), "r"(take ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LEFT>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory");
}

// ROWS x T tile at src (row stride as, first column col0) into shared memory;
// columns from ncol on read as zero.
template <int ROWS, int T, int THREADS>
__device__ __forceinline__ void tile_copy(float2* dst, const float2* src, long as, int col0, int ncol) {
  constexpr int CH = T / 2;
  for (int i = threadIdx.x; i < ROWS * CH; i += THREADS) {
    const int r = i / CH, c = 2 * (i % CH);
    const bool take = col0 + c < ncol;
    cp16(dst + r * T + c, take ? src + r * as + col0 + c : src, take);
  }
}

template <int N, int T, int SLOTS, int ROWS = N>
struct SpecSmem {
  AxisSmem<N> ax;
  float2 buf[Pencil<N, T, true>::BUF];
  alignas(16) float2 tile[SLOTS][ROWS * T];
};

template <int N, int T> using SpecPairSmem = SpecSmem<N, T, 2>;
template <int N, int T> using SpecISmem = SpecSmem<N, T, 1, spec_modes(N)>;

template <int N, int T>
constexpr int spec_min_blocks() {
  return (512 / (Shape<N>::A * T)) > 0 ? (512 / (Shape<N>::A * T)) : 1;
}

template <int N, int T>
__device__ __forceinline__ void tile_points(float2 (&v)[Shape<N>::B], const float2* tile, int t, int p) {
#pragma unroll
  for (int n2 = 0; n2 < Shape<N>::B; ++n2) v[n2] = tile[(t + Shape<N>::A * n2) * T + p];
}

// 3D y axis, forward: A = P G_x + D G_y and B = P G_z, masked modes dropped.
struct SpecFArgs {
  const float2* G;   // 3 wide arrays [plane][N][pitch]
  long gs;
  float2* out;       // A, then B at out + os: [plane][M][pitch]
  long os;
  int pitch, ncol;
  int planes, pps;   // planes of all solves, of one solve
  AxisOps ax;
  const int* active;
  int tile;          // columns per tile, 0: by rule
};

template <int N, int T>
__global__ void __launch_bounds__(Shape<N>::A * T, spec_min_blocks<N, T>()) k_spec_f(SpecFArgs a) {
  constexpr int A = Shape<N>::A, B = Shape<N>::B, M = spec_modes(N);
  using PF = Pencil<N, T, true>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  auto& S = *reinterpret_cast<SpecPairSmem<N, T>*>(smem_raw);
  load_axis<N>(S.ax, a.ax);
  dep_wait();
  const int p = threadIdx.x % T, t = threadIdx.x / T;
  PF pf{p, t, S.buf, S.ax.twf, S.ax.twi};
  const int ctiles = (a.ncol + T - 1) / T;
  const int items = ctiles * a.planes;
  // first item from w on whose solve is active
  auto next = [&](int w) {
    if (a.active != nullptr)
      while (w < items && a.active[w / ctiles / a.pps] == 0) w += gridDim.x;
    return w;
  };
  auto fetch = [&](int slot, int w, int f) {
    if (w < items)
      tile_copy<N, T, A * T>(S.tile[slot], a.G + f * a.gs + (long)(w / ctiles) * N * a.pitch, a.pitch,
                             (w % ctiles) * T, a.ncol);
    cp_commit();
  };
  int w = next(blockIdx.x);
  int s = 0;  // slot of the item's first tile
  fetch(0, w, 0);
  fetch(1, w, 1);
  while (w < items) {
    const int col = (w % ctiles) * T + p;
    const bool valid = col < a.ncol;
    float2* out = a.out + (long)(w / ctiles) * M * a.pitch + col;
    const int wn = next(w + gridDim.x);
    float2 v0[B], v1[B];
    cp_wait<0>();
    __syncthreads();
    tile_points<N, T>(v0, S.tile[s], t, p);
    tile_points<N, T>(v1, S.tile[s ^ 1], t, p);
    __syncthreads();
    fetch(s, w, 2);
    fetch(s ^ 1, wn, 0);
    pf.fwd(v0);
    pf.fwd(v1);
    sfor<0, B>([&](auto rc) {
      constexpr int r = decltype(rc)::value;
      if constexpr (spec_keeps<N>(r)) {
        const int k = pf.kidx(r);
        const int m = spec_col<N>(k);
        const float P = S.ax.P[k], d = S.ax.d[k];
        if (valid && m >= 0)
          out[(long)m * a.pitch] = make_float2(fmaf(P, v0[r].x, -d * v1[r].y), fmaf(P, v0[r].y, d * v1[r].x));
      }
    });
    cp_wait<1>();
    __syncthreads();
    tile_points<N, T>(v0, S.tile[s], t, p);
    __syncthreads();
    fetch(s, wn, 1);
    pf.fwd(v0);
    out += a.os;
    sfor<0, B>([&](auto rc) {
      constexpr int r = decltype(rc)::value;
      if constexpr (spec_keeps<N>(r)) {
        const int k = pf.kidx(r);
        const int m = spec_col<N>(k);
        const float P = S.ax.P[k];
        if (valid && m >= 0) out[(long)m * a.pitch] = make_float2(P * v0[r].x, P * v0[r].y);
      }
    });
    w = wn;
    s ^= 1;
  }
  cp_wait<0>();
}

// Last axis: k = -(P a + D b), RK bookkeeping in spectral space, increment
// back along the axis.  RK4: the accumulator holds sum_i w_i k_i of the
// stages so far; stages 0..2 return wnext k, stage 3 returns the whole
// increment of the step (rk_update_incr's weights).
struct SpecCArgs {
  const float2* a;   // P operand; [solve][outer][N][..] with the strides below
  const float2* b;   // D operand
  float2* out;       // increment; may alias a
  float2* acc;       // accumulator [solve][M][outer][..] (strides acc_as, acc_os)
  long as, os, ss;   // axis, outer and solve strides (complex elements)
  long acc_as, acc_os, acc_ss;
  int ncol, nouter, nsolve;
  AxisOps ax;
  int stage;         // 0..3
  int rk2;
  const double* dt_dev;
  double dt;
  const int* active;
  int tile;          // columns per tile, 0: by rule
};

template <int N, int T>
__global__ void __launch_bounds__(Shape<N>::A * T, spec_min_blocks<N, T>()) k_spec_c(SpecCArgs a) {
  constexpr int A = Shape<N>::A, B = Shape<N>::B;
  using PF = Pencil<N, T, true>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  auto& S = *reinterpret_cast<SpecPairSmem<N, T>*>(smem_raw);
  load_axis<N>(S.ax, a.ax);
  dep_wait();
  const int p = threadIdx.x % T, t = threadIdx.x / T;
  PF pf{p, t, S.buf, S.ax.twf, S.ax.twi};
  const int ctiles = (a.ncol + T - 1) / T;
  const int items = ctiles * a.nouter * a.nsolve;
  auto next = [&](int w) {
    if (a.active != nullptr)
      while (w < items && a.active[w / ctiles / a.nouter] == 0) w += gridDim.x;
    return w;
  };
  auto base_of = [&](int w) {
    const int o = w / ctiles;
    return (long)(o / a.nouter) * a.ss + (long)(o % a.nouter) * a.os;
  };
  auto fetch = [&](int w) {
    if (w < items) {
      const long b = base_of(w);
      tile_copy<N, T, A * T>(S.tile[0], a.a + b, a.as, (w % ctiles) * T, a.ncol);
      tile_copy<N, T, A * T>(S.tile[1], a.b + b, a.as, (w % ctiles) * T, a.ncol);
    }
    cp_commit();
  };
  int w = next(blockIdx.x);
  fetch(w);
  while (w < items) {
    const int col = (w % ctiles) * T + p;
    const int outer = w / ctiles % a.nouter, sol = w / ctiles / a.nouter;
    const bool valid = col < a.ncol;
    const int wn = next(w + gridDim.x);
    const float dt = (a.dt_dev != nullptr) ? (float)a.dt_dev[sol] : (float)a.dt;
    const RKCoef rk = rk_coef(a.stage, dt, a.rk2);
    float2* acc = a.acc + (long)sol * a.acc_ss + (long)outer * a.acc_os + col;
    float2 v[B], z2[B];
    cp_wait<0>();
    __syncthreads();
    tile_points<N, T>(v, S.tile[0], t, p);
    tile_points<N, T>(z2, S.tile[1], t, p);
    __syncthreads();
    fetch(wn);
    if (a.stage != 0 && valid) {  // the accumulator's lines, needed after the transforms
      sfor<0, B>([&](auto rc) {
        constexpr int r = decltype(rc)::value;
        if constexpr (spec_keeps<N>(r)) {
          const int m = spec_col<N>(pf.kidx(r));
          if (m >= 0 && p % 16 == 0) asm volatile("prefetch.global.L2 [%0];" ::"l"(acc + m * a.acc_as));
        }
      });
    }
    pf.fwd(v);
    pf.fwd(z2);
    sfor<0, B>([&](auto rc) {
      constexpr int r = decltype(rc)::value;
      if constexpr (spec_keeps<N>(r)) {
        const int k = pf.kidx(r);
        const float P = -S.ax.P[k], d = -S.ax.d[k];
        v[r] = make_float2(fmaf(P, v[r].x, -d * z2[r].y), fmaf(P, v[r].y, d * z2[r].x));
      }
    });
    // all of the accumulator's points in flight before the first is used: with
    // each load behind the previous point's store the thread waited for up to
    // B cache round trips in turn
    float2 (&q)[B] = z2;
    sfor<0, B>([&](auto rc) {
      constexpr int r = decltype(rc)::value;
      if constexpr (spec_keeps<N>(r)) {
        const int m = spec_col<N>(pf.kidx(r));
        q[r] = (a.stage != 0 && valid && m >= 0) ? acc[m * a.acc_as] : make_float2(0.0f, 0.0f);
      }
    });
    sfor<0, B>([&](auto rc) {
      constexpr int r = decltype(rc)::value;
      float2 inc = make_float2(0.0f, 0.0f);
      if constexpr (spec_keeps<N>(r)) {
        const int m = spec_col<N>(pf.kidx(r));
        if (m >= 0) {
          q[r] = make_float2(fmaf(rk.wacc, v[r].x, q[r].x), fmaf(rk.wacc, v[r].y, q[r].y));
          if (a.stage == 3) {
            inc = q[r];
          } else {
            if (valid) acc[m * a.acc_as] = q[r];
            inc = make_float2(rk.wnext * v[r].x, rk.wnext * v[r].y);
          }
        }
      }
      v[r] = inc;
    });
    pf.inv(v);
    if (valid) {
      float2* out = a.out + base_of(w) + (long)t * a.as + col;
#pragma unroll
      for (int n2 = 0; n2 < B; ++n2) out[(long)(A * n2) * a.as] = v[n2];
    }
    w = wn;
  }
  cp_wait<0>();
}

// 3D: inverse y transform of the increment, [plane][M][pitch] -> wide rows.
struct SpecIArgs {
  const float2* in;
  float2* D;          // [plane][N][pitch]
  int pitch, ncol;
  int planes, pps;
  AxisOps ax;
  const int* active;
  int tile;           // columns per tile, 0: by rule
};

template <int N, int T>
__global__ void __launch_bounds__(Shape<N>::A * T, spec_min_blocks<N, T>()) k_spec_i(SpecIArgs a) {
  constexpr int A = Shape<N>::A, B = Shape<N>::B, M = spec_modes(N);
  using PF = Pencil<N, T, true>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  auto& S = *reinterpret_cast<SpecISmem<N, T>*>(smem_raw);
  load_axis<N>(S.ax, a.ax);
  dep_wait();
  const int p = threadIdx.x % T, t = threadIdx.x / T;
  PF pf{p, t, S.buf, S.ax.twf, S.ax.twi};
  const int ctiles = (a.ncol + T - 1) / T;
  const int items = ctiles * a.planes;
  auto next = [&](int w) {
    if (a.active != nullptr)
      while (w < items && a.active[w / ctiles / a.pps] == 0) w += gridDim.x;
    return w;
  };
  auto fetch = [&](int w) {
    if (w < items)
      tile_copy<M, T, A * T>(S.tile[0], a.in + (long)(w / ctiles) * M * a.pitch, a.pitch, (w % ctiles) * T, a.ncol);
    cp_commit();
  };
  int w = next(blockIdx.x);
  fetch(w);
  while (w < items) {
    const int col = (w % ctiles) * T + p;
    const int wn = next(w + gridDim.x);
    float2 v[B];
    cp_wait<0>();
    __syncthreads();
    sfor<0, B>([&](auto rc) {
      constexpr int r = decltype(rc)::value;
      v[r] = make_float2(0.0f, 0.0f);
      if constexpr (spec_keeps<N>(r)) {
        const int m = spec_col<N>(pf.kidx(r));
        if (m >= 0) v[r] = S.tile[0][m * T + p];
      }
    });
    __syncthreads();
    fetch(wn);
    pf.inv(v);
    if (col < a.ncol) {
      float2* out = a.D + ((long)(w / ctiles) * N + t) * a.pitch + col;
#pragma unroll
      for (int n2 = 0; n2 < B; ++n2) out[(long)(A * n2) * a.pitch] = v[n2];
    }
    w = wn;
  }
  cp_wait<0>();
}

template <int N, int PHYS> cudaError_t launch_spec_x(int nd, bool inc, bool flux, const SpecXArgs& a, cudaStream_t s);
template <int N> cudaError_t launch_spec_f(const SpecFArgs& a, cudaStream_t s);
template <int N> cudaError_t launch_spec_c(const SpecCArgs& a, cudaStream_t s);
template <int N> cudaError_t launch_spec_i(const SpecIArgs& a, cudaStream_t s);

}  // namespace ps

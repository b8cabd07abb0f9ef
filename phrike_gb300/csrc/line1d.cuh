// 1D Fourier Euler on power-of-two grids: whole RK steps of a solve in one
// CTA, built for latency (k_line1d).  Semantics as k_step1d (euler1d.cuh),
// which stays for artificial viscosity.
//
// A 1D solve is one dependent chain of 4 right-hand sides and a filter per
// step, so its time is the latency of the transforms, not their arithmetic.
// k_step1d gives a pencil N/16 threads of 16 points: at N = 1024 two warps
// walk through 24 transforms of ~460 instructions one after the other (70 us
// per step).  Here N/4 threads hold 4 points each and both packed transforms
// ((rho, momentum) and energy) run together, two independent radix-4
// butterflies per thread and pass:
//   * forward decimation in frequency, inverse decimation in time, in place:
//     no reordering; the last forward and the first inverse pass are one
//     (radix 4 or 8), with the symbol applied in digit-reversed order between
//     them;
//   * the first pass's butterfly of a thread is its own 4 points, so fluxes
//     enter and increments leave the transform in registers, and the state,
//     the stage input and the accumulator never leave them;
//   * twiddles and symbols depend on the thread and the pass only and are
//     loaded once per launch;
//   * both applications of the end-of-step filter (inside the step and by
//     cadence, solver.py:119-120, 265-267) are one round trip with the symbol
//     of their product;
//   * the float64 time-step control runs on a warp of its own while the others
//     evaluate the first stage, which does not need dt.
// Bound now by shared-memory traffic and the exchange latency: 10.3 us per
// step at N = 1024 (before: 71), 5.4 at 256 (37), 72 at 4096 (214), the same
// for one solve and for 152.
#pragma once
#include "euler1d.cuh"

namespace ps {

template <int N>
struct Line {
  static_assert(N >= 16, "at least one pass beside the fused one");
  static constexpr int TH = N / 4;  // threads that hold points
  static constexpr int NP = (ilog2(N) - 2) / 2;  // radix-4 passes with an exchange after them (lengths > 8)
  static constexpr int RF = N >> (2 * NP);        // radix of the fused middle pass: 4 or 8
  static constexpr bool WARP = TH <= 32;          // all points in one warp
  static constexpr bool HELP = TH > 32 && TH < 1024;  // a warp for the time-step control
  static constexpr int BLOCK = (TH < 32 ? 32 : TH) + (HELP ? 32 : 0);
  static constexpr bool STATE_SMEM = N >= 2048;   // 544 and 1024 threads: 96 and 64 registers each
  static constexpr bool TW_SMEM = N >= 2048;
};

template <int N>
struct LineSmem {
  float2 buf[2][N];
  float2 tw[Line<N>::TW_SMEM ? N : 1];
  float un[Line<N>::STATE_SMEM ? 3 * N : 1];
  float acc[Line<N>::STATE_SMEM ? 3 * N : 1];
  float red[32];
  float dt;
  int stop;
};

// Bank swizzle of a transform buffer (16 float2 per 128-byte row): accesses
// with strides 1, 4 and >= 16 all cover the banks once per half warp.
__device__ __forceinline__ int line_swz(int i) { return i ^ (((i >> 4) & 3) * 5); }

template <bool INV>
__device__ __forceinline__ void radix4(float2& a, float2& b, float2& c, float2& d) {
  const float2 t0 = cadd(a, c), t1 = csub(a, c), t2 = cadd(b, d), e = csub(b, d);
  const float2 t3 = INV ? make_float2(-e.y, e.x) : make_float2(e.y, -e.x);
  a = cadd(t0, t2);
  c = csub(t0, t2);
  b = cadd(t1, t3);
  d = csub(t1, t3);
}

// Euler fluxes and steps of one CTA; see k_line1d.
template <int N>
struct LineFft {
  using Ln = Line<N>;
  static constexpr int TH = Ln::TH, NP = Ln::NP, RF = Ln::RF;
  LineSmem<N>& S;
  const int tid;
  const bool own;  // holds points
  float2 tw[Ln::TW_SMEM ? 1 : NP][3];
  float ds[RF], fs[RF];  // derivative and filter symbols of the fused pass's outputs

  __device__ __forceinline__ void sync() const {
    if constexpr (Ln::WARP) __syncwarp();
    else asm volatile("bar.sync 1, %0;" ::"n"(TH) : "memory");
  }
  static constexpr int len(int p) { return N >> (2 * p); }
  __device__ __forceinline__ int base(int p) const {
    const int m = len(p) / 4;
    return (tid / m) * len(p) + tid % m;
  }
  __device__ __forceinline__ float2 twiddle(int p, int q) const {
    if constexpr (Ln::TW_SMEM) return S.tw[(tid % (len(p) / 4)) * q * (N / len(p))];
    else return tw[p][q - 1];
  }

  // twiddles of the thread from W_N^k (natural order) and its symbols
  __device__ __forceinline__ void setup(const float2* w, const AxisOps& ax) {
    if (!Ln::TW_SMEM && own) {
      sfor<0, NP>([&](auto pc) {
        constexpr int p = decltype(pc)::value;
#pragma unroll
        for (int q = 1; q < 4; ++q) tw[p][q - 1] = w[(tid % (len(p) / 4)) * q * (N / len(p))];
      });
    }
#pragma unroll
    for (int q = 0; q < RF; ++q) {
      // position of the fused pass's output -> frequency (digits reversed)
      int pos = (RF == 4) ? 4 * (tid % TH) + q : 8 * (tid % (N / 8)) + q;
      int k = 0, w4 = 1;
      for (int L = N; L > RF; L /= 4) {
        const int m = L / 4;
        k += w4 * (pos / m);
        pos %= m;
        w4 *= 4;
      }
      k += w4 * pos;
      ds[q] = ax.d[k];
      fs[q] = (1.0f / N) - ax.P[k];
    }
  }

  // v[f][q]: points tid + q N/4 of the two transforms.  op 0: v <- -D v;
  // op 1: v <- C v, the complement of the filter; op 2: of the filter twice.
  __device__ __forceinline__ void round_trip(float2 (&v)[2][4], int op) {
    sfor<0, NP>([&](auto pc) {
      constexpr int p = decltype(pc)::value;
      constexpr int m = len(p) / 4;
      if (own) {
        const int b = base(p);
#pragma unroll
        for (int f = 0; f < 2; ++f) {
          if constexpr (p > 0) {
#pragma unroll
            for (int q = 0; q < 4; ++q) v[f][q] = S.buf[f][line_swz(b + q * m)];
          }
          radix4<false>(v[f][0], v[f][1], v[f][2], v[f][3]);
#pragma unroll
          for (int q = 1; q < 4; ++q) v[f][q] = cmul(v[f][q], twiddle(p, q));
#pragma unroll
          for (int q = 0; q < 4; ++q) S.buf[f][line_swz(b + q * m)] = v[f][q];
        }
      }
      sync();
    });
    auto symbol = [&](float2 x, int q) {
      if (op == 0) return make_float2(x.y * ds[q], -x.x * ds[q]);
      const float c = fs[q];
      const float s = (op == 1) ? c : c * (2.0f - (float)N * c);
      return make_float2(x.x * s, x.y * s);
    };
    if (own) {
      if constexpr (RF == 4) {
#pragma unroll
        for (int f = 0; f < 2; ++f) {
          float2 x[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) x[q] = S.buf[f][line_swz(4 * tid + q)];
          radix4<false>(x[0], x[1], x[2], x[3]);
#pragma unroll
          for (int q = 0; q < 4; ++q) x[q] = symbol(x[q], q);
          radix4<true>(x[0], x[1], x[2], x[3]);
#pragma unroll
          for (int q = 0; q < 4; ++q) S.buf[f][line_swz(4 * tid + q)] = x[q];
        }
      } else {  // N/8 butterflies per transform: one per thread
        float2* buf = S.buf[tid / (N / 8)];
        const int j = 8 * (tid % (N / 8));
        float2 x[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) x[q] = buf[line_swz(j + q)];
        dft<8, false>(x);
#pragma unroll
        for (int q = 0; q < 8; ++q) x[q] = symbol(x[q], q);
        dft<8, true>(x);
#pragma unroll
        for (int q = 0; q < 8; ++q) buf[line_swz(j + q)] = x[q];
      }
    }
    sync();
    sfor<0, NP>([&](auto pc) {
      constexpr int p = NP - 1 - decltype(pc)::value;
      constexpr int m = len(p) / 4;
      if (own) {
        const int b = base(p);
#pragma unroll
        for (int f = 0; f < 2; ++f) {
#pragma unroll
          for (int q = 0; q < 4; ++q) v[f][q] = S.buf[f][line_swz(b + q * m)];
#pragma unroll
          for (int q = 1; q < 4; ++q) v[f][q] = cmulc(v[f][q], twiddle(p, q));
          radix4<true>(v[f][0], v[f][1], v[f][2], v[f][3]);
          if constexpr (p > 0) {
#pragma unroll
            for (int q = 0; q < 4; ++q) S.buf[f][line_swz(b + q * m)] = v[f][q];
          }
        }
      }
      if constexpr (p > 0) sync();
    });
  }
};

template <int N>
__global__ void __launch_bounds__(Line<N>::BLOCK) k_line1d(Step1DArgs a, const float2* tw) {
  using Ln = Line<N>;
  constexpr int TH = Ln::TH;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  auto& S = *reinterpret_cast<LineSmem<N>*>(smem_raw);
  const int sol = blockIdx.x;
  const int tid = threadIdx.x;
  LineFft<N> ft{S, tid, tid < TH};
  if (!Ln::HELP || tid < TH) ft.setup(tw, a.ax);
  if constexpr (Ln::TW_SMEM) {
    for (int k = tid; k < N; k += blockDim.x) S.tw[k] = tw[k];
  }
  dep_wait();
  if (a.active != nullptr && a.active[sol] == 0) return;
  const bool cfl = a.t != nullptr;
  float* U = a.U + (long)sol * a.solve_stride;
  const float er = U[2 * N];  // E_ref; U is written only after the last step
  const float g1 = a.gamma - 1.0f;
  double tl = 0.0, te = 0.0;
  int taken = 0;
  // dt of the step from the block's wave speed (solver.py:384-417)
  auto control = [&](float speed) {
    const bool stop = !(tl < te - 1e-12);
    double d = (speed <= 0.0f) ? 1e-6 : (double)a.cfl * (double)a.dx / (double)speed;
    d = fmin(d, te - tl);
    S.dt = (float)d;
    S.stop = stop ? 1 : 0;
    if (!stop) {
      tl += d;
      ++taken;
    }
    return stop;
  };
  if (cfl && (Ln::HELP ? tid == TH : tid == 0)) {
    tl = a.t[sol];
    te = a.tend[sol];
  }
  // er is read by every thread before any writes U
  __syncthreads();

  if (Ln::HELP && tid >= TH) {  // the time-step warp
    if (!cfl) return;
    for (int step = 0; step < a.nsteps; ++step) {
      asm volatile("bar.sync 2, %0;" ::"n"(TH + 32) : "memory");
      int stop = 0;
      if (tid == TH) {
        float m = 0.0f;
        for (int w = 0; w < TH / 32; ++w) m = fmaxf(m, S.red[w]);
        stop = control(m);
      }
      stop = __shfl_sync(0xffffffffu, stop, 0);
      __threadfence_block();
      asm volatile("bar.arrive 3, %0;" ::"n"(TH + 32) : "memory");
      if (stop) break;
    }
    if (tid == TH) {
      a.t[sol] = tl;
      if (a.steps_done != nullptr) a.steps_done[sol] += taken;
    }
    return;
  }

  const bool own = tid < TH;
  const float pmin_shift = a.p_min - g1 * er;
  const float href = a.gamma * er;
  float un_r[3][4], acc_r[3][4], us[3][4];
  // state slots: registers, or this thread's shared-memory slots
  auto UN = [&](int c, int q) -> float& { return Ln::STATE_SMEM ? S.un[(c * 4 + q) * TH + tid] : un_r[c][q]; };
  auto AC = [&](int c, int q) -> float& { return Ln::STATE_SMEM ? S.acc[(c * 4 + q) * TH + tid] : acc_r[c][q]; };
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      float v = own ? U[c * N + tid + q * TH] : 1.0f;  // (a zero numerator takes the divide's slow path)
      if (c == 2 && own) v -= er;
      us[c][q] = v;
      if (own) {
        UN(c, q) = v;
        AC(c, q) = 0.0f;
      }
    }
  const int cad0 = (cfl && a.steps_done != nullptr) ? a.steps_done[sol] : a.step_counter0;
  float dt = (a.dt_dev != nullptr) ? (float)a.dt_dev[sol] : (float)a.dt;

#pragma unroll 1
  for (int step = 0; step < a.nsteps; ++step) {
    if (cfl) {  // wave speed of the state at the start of the step
      float sm = 0.0f;
      if (own) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float rho = us[0][q];
          const float u = us[1][q] / rho;
          const float pp = g1 * (us[2][q] - 0.5f * rho * u * u) + g1 * er;  // true pressure
          sm = fmaxf(sm, fabsf(u) + sqrtf(a.gamma * pp / rho));
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) sm = fmaxf(sm, __shfl_xor_sync(0xffffffffu, sm, o));
      if (tid % 32 == 0) S.red[tid / 32] = sm;
      if constexpr (Ln::HELP) {
        __threadfence_block();
        asm volatile("bar.arrive 2, %0;" ::"n"(TH + 32) : "memory");
      } else {
        ft.sync();
        if (tid == 0) {
          float m = 0.0f;
          for (int w = 0; w < (TH + 31) / 32; ++w) m = fmaxf(m, S.red[w]);
          control(m);
        }
        ft.sync();
      }
    }
    bool stop = false;
#pragma unroll 1
    for (int stage = 0; stage < 4; ++stage) {
      if (a.rk2 && (stage == 1 || stage == 2)) continue;
      float2 v[2][4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float rho = us[0][q], m = us[1][q], E = us[2][q];
        const float u = m / rho;
        const float p = g1 * (E - 0.5f * rho * u * u);  // p' (E holds E')
        const float mom = rho * u;
        v[0][q] = make_float2(mom, mom * u + p);
        v[1][q] = make_float2(((E + p) + href) * u, 0.0f);
      }
      ft.round_trip(v, 0);
      if (cfl && stage == 0) {
        if constexpr (Ln::HELP) asm volatile("bar.sync 3, %0;" ::"n"(TH + 32) : "memory");
        stop = S.stop != 0;
        if (stop) break;
        dt = S.dt;
      }
      const RKCoef rc = rk_coef(stage, dt, a.rk2);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        float k[3] = {v[0][q].x, v[0][q].y, v[1][q].x};
        if (a.gx != 0.0f) {  // gravity source (solver.py:82-91)
          const float rho = us[0][q];
          const float u = us[1][q] / rho;
          k[1] += rho * a.gx;
          k[2] += rho * a.gx * u;
        }
        float u3[3];
        if (own) {
#pragma unroll
          for (int c = 0; c < 3; ++c) u3[c] = rk_update_incr(stage, rc, k[c], UN(c, q), AC(c, q));
          clamp_state<1>(u3, a.gamma, a.rho_min, pmin_shift);
#pragma unroll
          for (int c = 0; c < 3; ++c) us[c][q] = u3[c];
        }
      }
    }
    if (stop) break;
    // end of step: filter inside the RK step, and again by cadence
    const bool second = ((cad0 + step) % a.filter_interval) == 0;
    float2 v[2][4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      v[0][q] = make_float2(us[0][q], us[1][q]);
      v[1][q] = make_float2(us[2][q], 0.0f);
    }
    ft.round_trip(v, second ? 2 : 1);
    if (own) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        us[0][q] -= v[0][q].x;
        us[1][q] -= v[0][q].y;
        us[2][q] -= v[1][q].x;
#pragma unroll
        for (int c = 0; c < 3; ++c) UN(c, q) = us[c][q];
      }
    }
  }
  if (!Ln::HELP && cfl && tid == 0) {
    a.t[sol] = tl;
    if (a.steps_done != nullptr) a.steps_done[sol] += taken;
  }
  if (own) {
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int q = 0; q < 4; ++q) U[c * N + tid + q * TH] = UN(c, q) + (c == 2 ? er : 0.0f);
  }
}

}  // namespace ps

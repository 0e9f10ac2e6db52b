// gs_split.cuh -- dense output and reverse passes split over threads where one thread per
// trajectory leaves the chip idle: small batches and the few long trajectories of uneven ones
// (float64; the saved states of every field with one thread per trajectory, the reverse pass
// for states of up to 3 components).
//
// A trajectory's integration is a serial chain, but with its checkpoints recorded the work
// around that chain is not:
//   * saveat_states_kernel: a requested time needs the checkpoint before it, up to K - 1 replay
//     steps and one re-step.  Each thread takes kPoints consecutive times of one trajectory,
//     instead of one lane of the forward taking them one by one while its warp waits.
//   * saveat_vjp_kernel: the VJPs of those re-steps (the cotangents they add to the bracketing
//     step's start state, and their parameter gradients), the same way, into a workspace.
//   * adjoint_split_kernel: the reverse pass is linear in the cotangent, so G lanes of a warp
//     take a G-th of the trajectory's steps each and run the step VJPs for the D unit
//     cotangents at the end of their part (and, with dense output, one more column that starts
//     at 0 and collects the re-steps' cotangents); the parts are then applied in sequence to
//     the true cotangent by shuffles.  The D (+ 1) columns share the step's forward
//     quantities and are independent of each other.  D (+ 1) VJPs per step instead of one, for
//     a chain G times shorter.
// Step boundaries of the parts depend on the trajectory's step count and G alone, and the
// states on neither K nor G, so gradients do not depend on the checkpoint interval or on which
// other trajectories share the batch, at one G; another G, and one thread per trajectory, are
// other evaluation orders of the same sums (gsolve.h says how far they agree).
//
// B200, stiff Van der Pol batch (20,011 trajectories, 2269 steps on average, 17,220 the longest,
// 64 saved times): reverse pass 8.9 ms with one lane each, 2.25 ms with 16.
#pragma once
#include <math_constants.h>

#include "gs_persistent.cuh"
#include "gs_saveat.cuh"

namespace gs {

constexpr int kSplitMaxDim = 3;
constexpr int kPoints = 4;  // consecutive requested times per thread of the saveat kernels

// The forward quantities of one step, shared by the columns' VJPs.
struct Tsit5Split {
  using Step = Tsit5F64Step;
  static constexpr bool kRefine = false;
  template <class F>
  struct Fwd {
    StageStates<F> S;
  };
  template <class F>
  static __device__ __forceinline__ void prepare(const double* y, const double* p, double dt,
                                                 Fwd<F>& f) {
    tsit5_stage_states<F, false>(y, p, dt, f.S, static_cast<double*>(nullptr));
  }
  template <class F>
  static __device__ __forceinline__ void vjp(const double* y, const double* p, double dt,
                                             const Fwd<F>& f, double* lam, double* gp) {
    tsit5_vjp_core<F>(y, f.S, p, dt, lam, gp);
  }
};

struct Ros23Split {
  using Step = Ros23Step;
  static constexpr bool kRefine = true;
  template <class F>
  struct Fwd {
    RosCore<F> c;
    double s1[F::D];
  };
  template <class F>
  static __device__ __forceinline__ void prepare(const double* y, const double* p, double dt,
                                                 Fwd<F>& f) {
    double yn[F::D];
    ros23_core<F>(y, p, dt, f.c, yn);
#pragma unroll
    for (int i = 0; i < F::D; ++i) f.s1[i] = y[i] + 0.5 * dt * f.c.k1[i];
  }
  template <class F>
  static __device__ __forceinline__ void vjp(const double* y, const double* p, double dt,
                                             const Fwd<F>& f, double* lam, double* gp) {
    ros23_vjp_core<F>(y, p, dt, f.c.W, f.c.k1, f.s1, f.c.k2p, lam, gp);
  }
};

// ---- requested times from the checkpoints -------------------------------------------------
// A walk along trajectory j's recorded steps from its checkpoints: seek(ts) moves to the step
// that brackets ts (t < ts <= t + dt, t its start), or to the end of the record.
template <class F, class M>
struct StepWalk {
  static constexpr int D = F::D, CW = (D + 2) & ~1;
  const SaveatArgs& a;
  long long j;
  int na, slots, s, c;  // steps; checkpoint slots written; current step; its slot
  double y[D], t, dt;

  __device__ __forceinline__ StepWalk(const SaveatArgs& args, long long jj)
      : a(args), j(jj), na(steps_in_record(args.n_acc, jj, args.cap)), s(0), c(-1), t(0.0),
        dt(0.0) {
    const int w = na / a.ck_every + 1;
    slots = w < a.ck_slots ? w : a.ck_slots;
  }
  __device__ __forceinline__ double slot_time(int k) const {
    return __ldg(a.ckpt + ((size_t)k * (size_t)a.n + (size_t)j) * CW + D);
  }
  // true: step s at state y, time t, of size dt, brackets ts; false: no step does.  ts > t0,
  // and not below the last call's.
  __device__ __forceinline__ bool seek(double ts, const double* p) {
    if (c < 0 || (c + 1 < slots && slot_time(c + 1) < ts)) {
      int lo = c < 0 ? 0 : c + 1, hi = slots;  // slot_time(lo) < ts
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (slot_time(mid) < ts)
          lo = mid;
        else
          hi = mid;
      }
      c = lo;
      s = c * a.ck_every;
      t = load_ckpt<D>(a.ckpt, a.n, j, c, y);
    }
    for (; s < na; ++s) {
      dt = load_rec(a.rec, a.n, j, s);
      if (dt > 0.0) {
        const double tn = t + dt;
        if (ts <= tn) return true;
        double cy[D];
#pragma unroll
        for (int i = 0; i < D; ++i) cy[i] = 0.0;
        M::template step<F>(y, cy, p, nullptr, dt);
        t = tn;
      }
    }
    return false;
  }
  // whether the bracketing step is the last and ts its end: the final state itself
  __device__ __forceinline__ bool at_end(double ts) const { return s == na - 1 && ts >= t + dt; }
};

// ys of a recorded forward (rules: gs_saveat.cuh), from its record, checkpoints and y_final.
template <class F, class M>
__global__ void __launch_bounds__(128) saveat_states_kernel(const SaveatArgs a) {
  constexpr int D = F::D, P = F::P;
  const long long parts = (a.K + kPoints - 1) / kPoints;
  const long long u = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (u >= a.n * parts) return;
  const long long j = u / parts;
  const int k0 = (int)(u - j * parts) * kPoints;
  const int k1 = k0 + kPoints < a.K ? k0 + kPoints : a.K;
  double p[P];
#pragma unroll
  for (int i = 0; i < P; ++i) p[i] = a.p[j * P + i];
  const double* ts = a.ts + j * a.ts_ld;
  double* ys = a.ys + j * (long long)a.K * D;
  const double* yf = a.yf + j * D;
  StepWalk<F, M> w(a, j);
  for (int k = k0; k < k1; ++k) {
    const double tk = ts[k];
    double* dst = ys + (long long)k * D;
    if (tk <= a.t0) {  // never bracketed: y0 (y_final, the same, of a trajectory without steps)
      double y0[D];
      load_ckpt<D>(a.ckpt, a.n, j, 0, y0);
      store_row<D>(dst, y0);
    } else if (w.seek(tk, p) && !w.at_end(tk)) {
      double yk[D], cy[D];
#pragma unroll
      for (int i = 0; i < D; ++i) { yk[i] = w.y[i]; cy[i] = 0.0; }
      M::template step<F>(yk, cy, p, nullptr, tk - w.t);
      store_row<D>(dst, yk);
    } else {  // at or past the final accumulated time
#pragma unroll
      for (int i = 0; i < D; ++i) dst[i] = yf[i];
    }
  }
}

// The re-steps' VJPs: work row (j * K + k) of D + P values gets, for a bracketed time, the
// cotangent it adds to the bracketing step's start state and its parameter gradient (rows of
// other times are not written, and not read by adjoint_split_kernel).
template <class F, class M>
__global__ void __launch_bounds__(128) saveat_vjp_kernel(const SaveatArgs a, double* work) {
  constexpr int D = F::D, P = F::P;
  const long long parts = (a.K + kPoints - 1) / kPoints;
  const long long u = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (u >= a.n * parts) return;
  const long long j = u / parts;
  const int k0 = (int)(u - j * parts) * kPoints;
  const int k1 = k0 + kPoints < a.K ? k0 + kPoints : a.K;
  double p[P];
#pragma unroll
  for (int i = 0; i < P; ++i) p[i] = a.p[j * P + i];
  const double* ts = a.ts + j * a.ts_ld;
  StepWalk<F, M> w(a, j);
  const double t0 = w.slot_time(0);
  for (int k = k0; k < k1; ++k) {
    const double tk = ts[k];
    if (tk <= t0) continue;
    if (!w.seek(tk, p)) return;  // (later times lie past the end too)
    if (w.at_end(tk)) continue;
    const long long row = j * a.K + k;
    double v[D], gp[P];
#pragma unroll
    for (int i = 0; i < D; ++i) v[i] = a.ysbar[row * D + i];
#pragma unroll
    for (int i = 0; i < P; ++i) gp[i] = 0.0;
    M::template vjp<F>(w.y, p, nullptr, tk - w.t, v, gp);
#pragma unroll
    for (int i = 0; i < D; ++i) work[row * (D + P) + i] = v[i];
#pragma unroll
    for (int i = 0; i < P; ++i) work[row * (D + P) + D + i] = gp[i];
  }
}

// The recorded steps a pass takes: those of the replay whose checkpoints it reads.  Dense output
// walks forward in time (gs_saveat.cuh); the plain replay takes every step that is not 0, so a
// mesh given by the caller may also step backwards, and a NaN step makes the gradient NaN.
template <bool kSave>
__device__ __forceinline__ bool takes_step(double dt) {
  return kSave ? dt > 0.0 : dt != 0.0;
}

// ---- the split reverse pass ------------------------------------------------------------------
// One sweep of a lane's steps [lo, hi) of trajectory j, latest first: their VJPs applied to the C
// columns lam, gp; column C - 1 collects the re-steps' cotangents (kSave).  kfin: the number of
// requested times of this lane's part and the ones before it.
template <class F, class S, bool kSave, int C>
__device__ __forceinline__ void split_sweep(const SaveatArgs& a, const double* work, long long j,
                                            int na, int lo, int hi, const double* p,
                                            double (&lam)[C][F::D], double (&gp)[C][F::P],
                                            int& kfin) {
  constexpr int D = F::D, P = F::P;
  const int K = a.ck_every;
  // dense output: times [0, kk) not yet assigned; tlast = ts[kk - 1] (-inf without one)
  const double* ts = kSave ? a.ts + j * a.ts_ld : nullptr;
  int kk = 0;
  double tlast = -CUDART_INF;
  AdjBuf<D, D + 1> buf(K);
  int b = 0;
  const int top = hi > lo ? (hi - 1) / K : -1, bottom = lo / K;
  if (top >= 0) prefetch_segment<D>(buf, b, a.ckpt, a.rec, a.n, j, top, K, na);
  for (int sg = top; sg >= 0 && sg >= bottom; --sg) {
    cp_async_wait_all();
    double y[D];
#pragma unroll
    for (int i = 0; i < D; ++i) y[i] = buf.ck(b, i);
    double t = buf.ck(b, D);
    if (sg > bottom) prefetch_segment<D>(buf, b ^ 1, a.ckpt, a.rec, a.n, j, sg - 1, K, na);
    const int q1 = hi - sg * K < K ? hi - sg * K : K;   // this lane's steps of the segment:
    const int q0 = lo > sg * K ? lo - sg * K : 0;       // [q0, q1)
    for (int q = 0; q < q1; ++q) {  // states and times at the start of steps 0 .. q1 - 1
#pragma unroll
      for (int i = 0; i < D; ++i) buf.st(q, i) = y[i];
      buf.st(q, D) = t;
      const double dt = buf.dt(b, q);
      if (takes_step<kSave>(dt)) {
        if (q + 1 < q1) {
          double cy[D];
#pragma unroll
          for (int i = 0; i < D; ++i) cy[i] = 0.0;
          S::Step::template step<F>(y, cy, p, nullptr, dt);
        }
        t = t + dt;
      }
    }
    if (kSave && sg == top) {  // t: the end of this lane's part
      // times up to it, or strictly before it where it is the trajectory's end
      int x0 = 0, x1 = a.K;
      while (x0 < x1) {
        const int mid = (x0 + x1) >> 1;
        if (hi < na ? ts[mid] <= t : ts[mid] < t)
          x0 = mid + 1;
        else
          x1 = mid;
      }
      kk = kfin = x0;
      tlast = kk > 0 ? ts[kk - 1] : -CUDART_INF;
    }
    for (int q = q1 - 1; q >= q0; --q) {
      const double dt = buf.dt(b, q);
      if (takes_step<kSave>(dt)) {
        double ys[D];
#pragma unroll
        for (int i = 0; i < D; ++i) ys[i] = buf.st(q, i);
        const double ts0 = buf.st(q, D);
        typename S::template Fwd<F> f;
        S::template prepare<F>(ys, p, dt, f);
#pragma unroll
        for (int c = 0; c < C; ++c) S::template vjp<F>(ys, p, dt, f, lam[c], gp[c]);
        if constexpr (kSave) {
          while (tlast > ts0) {
            const double* row = work + (j * (long long)a.K + (kk - 1)) * (D + P);
#pragma unroll
            for (int i = 0; i < D; ++i) lam[C - 1][i] += row[i];
#pragma unroll
            for (int i = 0; i < P; ++i) gp[C - 1][i] += row[D + i];
            --kk;
            tlast = kk > 0 ? ts[kk - 1] : -CUDART_INF;
          }
        }
      }
    }
    b ^= 1;
  }
}

// G lanes (a power of two, at most 32) per trajectory; order: as AdjointArgs.  kSave: with the
// cotangents of dense output (a.ts, a.ysbar, work of saveat_vjp_kernel).
//
// S::kRefine: a second sweep with the cotangents that the composition found.  Over a part of a
// contracting (stiff) trajectory the columns are nearly parallel and the true cotangent may be
// nearly orthogonal to what they have in common, so their sum cancels: on stiff Van der Pol
// trajectories (17,000 steps, 8 lanes) rows were off by 5e-13 at the median and 2.6e-11 at most
// against 80-bit arithmetic, where one thread per trajectory is off by 5e-14 and 1.5e-12.  The
// second sweep runs each part from the cotangent at its end as one thread would; what it
// leaves at the part before differs from that part's cotangent by the cancelled digits, and the
// columns carry these differences through the parts: one thread's errors, for 1.6 to 1.9 times
// the pass (20,011 trajectories of 2269 steps on average, 16 lanes, K = 8: 1.05 / 1.73 ms, with 64
// saved times 1.32 / 2.25; one thread each, lanes refilled, 7.3 and 8.9).  Tsit5's trajectories
// are not stiff for it (its errors against 80-bit arithmetic are one thread's on Van der Pol and on
// Lorenz up to t = 70), and take one sweep.
template <class F, class S, bool kSave>
__global__ void __launch_bounds__(128) adjoint_split_kernel(const SaveatArgs a, int G,
                                                            const double* work,
                                                            const long long* order) {
  constexpr int D = F::D, P = F::P, C = D + (kSave ? 1 : 0);
  const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int l = (int)(threadIdx.x & (unsigned)(G - 1));
  long long j = tid / G;
  const bool live = j < a.n;
  if (!live) j = a.n - 1;  // (the lanes past the batch keep the warp's shuffles whole)
  if (order) {
    const long long o = __ldg(order + j);
    j = (o >= 0 && o < a.n) ? o : -1;
  }
  const bool idle = j < 0;  // an entry of order outside the batch
  if (idle) j = 0;
  double p[P];
#pragma unroll
  for (int i = 0; i < P; ++i) p[i] = a.p[j * P + i];
  const int na = live && !idle ? steps_in_record(a.n_acc, j, a.cap) : 0;
  const int lo = (int)((long long)na * l / G), hi = (int)((long long)na * (l + 1) / G);
  double lam[C][D], gp[C][P];
#pragma unroll
  for (int c = 0; c < C; ++c) {
#pragma unroll
    for (int i = 0; i < D; ++i) lam[c][i] = c == i ? 1.0 : 0.0;
#pragma unroll
    for (int i = 0; i < P; ++i) gp[c][i] = 0.0;
  }
  const double* ts = kSave ? a.ts + j * a.ts_ld : nullptr;
  const double* ysb = kSave ? a.ysbar + j * (long long)a.K * D : nullptr;
  int kfin = 0;  // (the last lane's: the times at or past the end, from there on)
  split_sweep<F, S, kSave>(a, work, j, na, lo, hi, p, lam, gp, kfin);
  // the cotangent at the trajectory's end, from its last lane, through the parts in sequence
  double cur[D], in[D];
#pragma unroll
  for (int i = 0; i < D; ++i) cur[i] = a.ybar ? a.ybar[j * D + i] : 0.0;
  if constexpr (kSave) {
    if (l == G - 1) {
      // (kfin = 0 without steps: every time is y_final = y0)
      for (int k = a.K - 1; live && !idle && k >= kfin; --k) {
#pragma unroll
        for (int i = 0; i < D; ++i) cur[i] += ysb[(long long)k * D + i];
      }
    }
  }
  const int base = (int)(threadIdx.x & 31u) & ~(G - 1);
#pragma unroll
  for (int i = 0; i < D; ++i) cur[i] = __shfl_sync(0xffffffffu, cur[i], base + G - 1);
#pragma unroll
  for (int i = 0; i < D; ++i) in[i] = cur[i];
  for (int m = G - 1; m >= 0; --m) {
    double out[D];
#pragma unroll
    for (int i = 0; i < D; ++i) {
      double v = lam[0][i] * cur[0];
#pragma unroll
      for (int c = 1; c < D; ++c) v = v + lam[c][i] * cur[c];
      if constexpr (kSave) v = v + lam[D][i];
      out[i] = v;
    }
    if (l == m) {
#pragma unroll
      for (int i = 0; i < D; ++i) in[i] = cur[i];
    }
#pragma unroll
    for (int i = 0; i < D; ++i) cur[i] = __shfl_sync(0xffffffffu, out[i], base + m);
  }
  double own[P];  // the part's share of the parameter gradient
  if constexpr (S::kRefine && D > 1) {  // (one component: nothing cancels)
    double v[1][D], g[1][P], e[D], in_e[D];
#pragma unroll
    for (int i = 0; i < D; ++i) v[0][i] = in[i];
#pragma unroll
    for (int i = 0; i < P; ++i) g[0][i] = 0.0;
    split_sweep<F, S, kSave>(a, work, j, na, lo, hi, p, v, g, kfin);
    // e: what the cotangent at a part's end lacks; the last part's is exact
#pragma unroll
    for (int i = 0; i < D; ++i) {
      const double after = __shfl_down_sync(0xffffffffu, v[0][i], 1);
      in_e[i] = l == G - 1 || after == in[i] ? 0.0 : after - in[i];
      e[i] = 0.0;
    }
    for (int m = G - 1; m >= 0; --m) {
#pragma unroll
      for (int i = 0; i < D; ++i) e[i] += __shfl_sync(0xffffffffu, in_e[i], base + m);
      if (l == m) {
#pragma unroll
        for (int i = 0; i < D; ++i) in_e[i] = e[i];
      }
      double out[D];
#pragma unroll
      for (int i = 0; i < D; ++i) {
        double x = lam[0][i] * e[0];
#pragma unroll
        for (int c = 1; c < D; ++c) x = x + lam[c][i] * e[c];
        out[i] = x;
      }
#pragma unroll
      for (int i = 0; i < D; ++i) e[i] = __shfl_sync(0xffffffffu, out[i], base + m);
    }
#pragma unroll
    for (int i = 0; i < D; ++i) cur[i] = v[0][i] + e[i];  // (of lane 0)
#pragma unroll
    for (int i = 0; i < P; ++i) {
      own[i] = g[0][i];
#pragma unroll
      for (int c = 0; c < D; ++c) own[i] = own[i] + gp[c][i] * in_e[c];
    }
  } else {
#pragma unroll
    for (int i = 0; i < P; ++i) {
      double v = gp[0][i] * in[0];
#pragma unroll
      for (int c = 1; c < D; ++c) v = v + gp[c][i] * in[c];
      if constexpr (kSave) v = v + gp[D][i];
      own[i] = v;
    }
  }
  if constexpr (kSave) kfin = __shfl_sync(0xffffffffu, kfin, base + G - 1);
#pragma unroll
  for (int i = 0; i < P; ++i) {
    double v = own[i];
    for (int o = 1; o < G; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (a.gp && l == 0 && live && !idle) a.gp[j * P + i] = v;
  }
  if (l == 0 && live && !idle) {
    if constexpr (kSave) {  // times at or before t0 take y0: their cotangents join dL/dy0
      const double t0 = a.ckpt[(size_t)j * ((D + 2) & ~1) + D];
      for (int k = 0; k < kfin && ts[k] <= t0; ++k) {
#pragma unroll
        for (int i = 0; i < D; ++i) cur[i] += ysb[(long long)k * D + i];
      }
    }
    if (a.gy0) {
#pragma unroll
      for (int i = 0; i < D; ++i) a.gy0[j * D + i] = cur[i];
    }
  }
}

}  // namespace gs

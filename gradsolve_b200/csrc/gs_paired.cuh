// gs_paired.cuh -- reverse pass with two warps per 32 trajectories (float64): for batches that
// leave each scheduler one or two warps of the one-thread kernels.
//
// A reverse step recomputes the step's forward quantities (Tsit5: its stage inputs;
// Rosenbrock23: the factors of W, k1, s1 and k2') and applies its VJP.  The first does not wait
// for the cotangent, so a block's first warp runs it for segment sg - 1 while the second applies
// the VJPs of segment sg; they hand segments over through a double buffer in shared memory, one
// block barrier per segment.  The same work on twice the warps, each with half the chain, and the
// same expressions (tsit5_stage_states, tsit5_vjp_core, ros23_core_as, ros23_vjp_core).
//
// Both warps run `top` + 1 rounds, top the segment count of the longest of the 32 trajectories
// (from the same step counts, so equal in both), and every thread reaches every barrier.
#pragma once

#include "gs_ros23.cuh"
#include "gs_tsit5.cuh"

namespace gs {

// One step in the buffer: the state, dt and the method's words; element e of lane l at e * 32 + l.
template <class F>
struct Tsit5Pair {
  static constexpr int D = F::D, kWords = 5 * D;
  static __device__ __forceinline__ void produce(const double* y, const double* p, double dt,
                                                 double* w, double* ynext, bool next) {
    StageStates<F> S;
    if (next)
      tsit5_stage_states<F, true>(y, p, dt, S, ynext);
    else
      tsit5_stage_states<F, false>(y, p, dt, S, ynext);
#pragma unroll
    for (int i = 0; i < D; ++i) {
      w[(0 * D + i) * 32] = S.s2[i];
      w[(1 * D + i) * 32] = S.s3[i];
      w[(2 * D + i) * 32] = S.s4[i];
      w[(3 * D + i) * 32] = S.s5[i];
      w[(4 * D + i) * 32] = S.s6[i];
    }
  }
  struct Source {
    const double* w;
    template <int M>
    __device__ __forceinline__ void get(double* out) const {
#pragma unroll
      for (int i = 0; i < D; ++i) out[i] = w[((M - 2) * D + i) * 32];
    }
  };
  static __device__ __forceinline__ void consume(const double* y, const double* p, double dt,
                                                 const double* w, double* lam, double* gp) {
    tsit5_vjp_core<F>(y, Source{w}, p, dt, lam, gp);
  }
};

template <class F>
struct Ros23Pair {
  static constexpr int D = F::D;
  static constexpr bool kSparse = kSparseW<F, double>;
  // W's entries (the sparse factors' nonzero ones), 1 / U's diagonal and the pivots (LU only),
  // k1, s1, k2' and, for a sparse W, whether its pivots hold
  static constexpr int kEntries = kSparse ? bit_count(kLU<F>) : D * D;
  static constexpr int kInv = kInverseW<D, double> ? 0 : D;
  static constexpr int kPiv = kInverseW<D, double> || kSparse ? 0 : D;
  static constexpr int kWords = kEntries + kInv + kPiv + 3 * D + (kSparse ? 1 : 0);

  template <class T, class Fn>
  static __device__ __forceinline__ void each(T* w, Fn fn) {  // fn(word, entry) over W's entries
    int k = 0;
#pragma unroll
    for (int e = 0; e < D * D; ++e) {
      if (!kSparse || ((kLU<F> >> e) & 1)) fn(w[32 * k++], e);
    }
  }
  static __device__ __forceinline__ void produce(const double* y, const double* p, double dt,
                                                 double* w, double* ynext, bool) {
    RosCore<F> c;
    const bool ok = ros23_core_as<F, kSparse>(y, p, dt, c, ynext);
    each(w, [&](double& word, int e) { word = c.W.a[e]; });
    w += 32 * kEntries;
    if constexpr (kInv > 0) {
#pragma unroll
      for (int i = 0; i < D; ++i) w[32 * i] = c.W.inv[i];
      w += 32 * kInv;
    }
    if constexpr (kPiv > 0) {
#pragma unroll
      for (int i = 0; i < D; ++i) w[32 * i] = (double)c.W.piv[i];
      w += 32 * kPiv;
    }
#pragma unroll
    for (int i = 0; i < D; ++i) {
      w[32 * i] = c.k1[i];
      w[32 * (D + i)] = y[i] + 0.5 * dt * c.k1[i];
      w[32 * (2 * D + i)] = c.k2p[i];
    }
    if constexpr (kSparse) {
      w[32 * 3 * D] = ok ? 1.0 : 0.0;
      if (!ok) from_dvec<D>(ros23_step_pivoted<F>(to_dvec<D>(y), to_dvec<F::P>(p), dt), ynext);
    }
  }
  static __device__ __forceinline__ void consume(const double* y, const double* p, double dt,
                                                 const double* w, double* lam, double* gp) {
    constexpr int P = F::P;
    if constexpr (kSparse) {
      if (w[32 * (kWords - 1)] == 0.0) {  // another pivot: the pivoted elimination, out of line
        const DVec<D + P> r = ros23_step_vjp_pivoted<F>(to_dvec<D>(y), to_dvec<P>(p), dt,
                                                        to_dvec<D>(lam), to_dvec<P>(gp));
#pragma unroll
        for (int i = 0; i < D; ++i) lam[i] = r.v[i];
#pragma unroll
        for (int i = 0; i < P; ++i) gp[i] = r.v[D + i];
        return;
      }
    }
    LU<D> W;
    double k1[D], s1[D], k2p[D];
    each(w, [&](const double& word, int e) { W.a[e] = word; });
    w += 32 * kEntries;
    if constexpr (kInv > 0) {
#pragma unroll
      for (int i = 0; i < D; ++i) W.inv[i] = w[32 * i];
      w += 32 * kInv;
    }
    if constexpr (kPiv > 0) {
#pragma unroll
      for (int i = 0; i < D; ++i) W.piv[i] = (int)w[32 * i];
      w += 32 * kPiv;
    }
#pragma unroll
    for (int i = 0; i < D; ++i) {
      k1[i] = w[32 * i];
      s1[i] = w[32 * (D + i)];
      k2p[i] = w[32 * (2 * D + i)];
    }
    ros23_vjp_core<F, double, kSparse>(y, p, dt, W, k1, s1, k2p, lam, gp);
  }
};

// Doubles of the two buffers per thread of the 64 (2 K steps of D + 1 + words, 32 lanes), and of
// the whole shared memory with the producers' prefetch area.
template <class F, class S>
GS_HD int paired_buffer_doubles(int K) { return K * (F::D + 1 + S::kWords); }
template <class F, class S>
GS_HD int paired_smem_doubles(int K) {
  return paired_buffer_doubles<F, S>(K) + seg_io_doubles<F::D>(K);
}

template <class F, class S>
__global__ void __launch_bounds__(64) adjoint_paired_kernel(const AdjointArgs a) {
  constexpr int D = F::D, P = F::P, WS = D + 1 + S::kWords;
  const int lane = threadIdx.x & 31;
  const bool producer = threadIdx.x < 32;
  const long long t = (long long)blockIdx.x * 32 + lane;
  long long j = t < a.n ? lane_traj(a, t) : -1;
  const bool live = j >= 0;
  if (!live) j = 0;
  double p[P];
#pragma unroll
  for (int i = 0; i < P; ++i) p[i] = a.p[j * P + i];
  const int na = live ? steps_in_record(a.n_acc, j, a.cap) : 0;
  const int K = a.ck_every;
  const int nseg = (na + K - 1) / K;
  const int top = __reduce_max_sync(0xffffffffu, nseg);
  // step q of buffer b: words at buf + ((b * K + q) * WS + e) * 32
  double* const buf = gs_seg_smem + lane;
  SegIO<D> io(paired_buffer_doubles<F, S>(K), K);
  struct {
    SegIO<D>& io;
  } fetch{io};
  double lam[D], gp[P];
#pragma unroll
  for (int i = 0; i < D; ++i) lam[i] = live ? a.ybar[j * D + i] : 0.0;
#pragma unroll
  for (int i = 0; i < P; ++i) gp[i] = 0.0;
  int b = 0;
  if (producer && nseg > 0) prefetch_segment<D>(fetch, b, a.ckpt, a.rec, a.n, j, nseg - 1, K, na);
  for (int it = 0; it <= top; ++it) {
    if (producer) {
      const int sg = top - 1 - it;
      if (it < top && sg < nseg) {
        cp_async_wait_all();
        double y[D];
#pragma unroll
        for (int i = 0; i < D; ++i) y[i] = io.ck(b, i);
        if (sg > 0) prefetch_segment<D>(fetch, b ^ 1, a.ckpt, a.rec, a.n, j, sg - 1, K, na);
        for (int q = 0; q < K; ++q) {
          double* const w = buf + ((it & 1) * K + q) * (WS * 32);
          const double dt = io.dt(b, q);
#pragma unroll
          for (int i = 0; i < D; ++i) w[32 * i] = y[i];
          w[32 * D] = dt;
          if (dt != 0.0) {
            double yn[D];
            S::produce(y, p, dt, w + 32 * (D + 1), yn, q + 1 < K);
            if (q + 1 < K) {
#pragma unroll
              for (int i = 0; i < D; ++i) y[i] = yn[i];
            }
          }
        }
        b ^= 1;
      }
    } else {
      const int sg = top - it;
      if (it > 0 && sg < nseg) {
        for (int q = K - 1; q >= 0; --q) {
          const double* const w = buf + (((it - 1) & 1) * K + q) * (WS * 32);
          const double dt = w[32 * D];
          if (dt != 0.0) {
            double y[D];
#pragma unroll
            for (int i = 0; i < D; ++i) y[i] = w[32 * i];
            S::consume(y, p, dt, w + 32 * (D + 1), lam, gp);
          }
        }
      }
    }
    __syncthreads();
  }
  if (!producer && live) {
    if (a.gy0) {
#pragma unroll
      for (int i = 0; i < D; ++i) a.gy0[j * D + i] = lam[i];
    }
    if (a.gp) {
#pragma unroll
      for (int i = 0; i < P; ++i) a.gp[j * P + i] = gp[i];
    }
  }
}

}  // namespace gs

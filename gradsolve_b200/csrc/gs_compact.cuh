// gs_compact.cuh -- recording forward of a fresh large batch that compacts its finished
// trajectories (float64 and float32-stage Tsit5, Rosenbrock23; states of up to 4 components).
//
// One thread integrates one trajectory, and a warp runs until its longest one ends: where the
// step counts spread (Robertson 370 to 1000 attempts, Lotka-Volterra 40 to 190) a third of the
// lanes idle.  A batch solved before is ordered by its counts; a fresh one is not.  So a warp
// whose active lanes fall below kKeep writes their states to a list in global memory and ends,
// and the next launch takes the list with full warps: kPasses launches, the last one to the end.
// The attempts, the record and the checkpoints are those of the one-thread kernels, trajectory by
// trajectory; the order in the lists depends on the run, what is computed does not.
#pragma once

#include "gs_mixed.cuh"
#include "gs_ros23.cuh"
#include "gs_tsit5.cuh"

namespace gs {

// B200, one launch / 12, 16, 20 lanes kept (3, 4, 4 launches): Robertson 2^18 3.22 / 2.75, 2.71,
// 2.68 ms, 2^17 1.73 / 1.54, 1.53, 1.51; Lotka-Volterra float32 stages 2^18 388 / 367, 374, 367 us,
// float64 2^18 428 / 397, 399, 397, 2^20 1538 / 1342, 1316, 1341; Lorenz (counts within 7%) 2^20
// 9.96 / 9.92, 9.92, 9.93 ms, 2^18 2.596 / 2.600, 2.606, 2.620.
constexpr int kKeep = 16;
constexpr int kPasses = 4;

// The state carried from attempt to attempt: kState doubles.
template <class F>
struct CompactTsit5 {
  static constexpr int D = F::D, kState = 2 * D, QK = 10;
  static __device__ __forceinline__ void begin(const double* y0, const double* p, double* s) {
#pragma unroll
    for (int i = 0; i < D; ++i) s[i] = y0[i];
    F::rhs(s, p, s + D);
  }
  static __device__ __forceinline__ bool attempt(const RecordArgs& a, long long j, const double* p,
                                                 const float*, double t1, long long rstride,
                                                 FwdCounters& c, const double* s, double* o) {
    return tsit5_attempt<F>(a, j, p, t1, true, true, rstride, c, s, s + D, o, o + D);
  }
};

template <class F>
struct CompactMixed {
  static constexpr int D = F::D, kState = 3 * D, QK = 10;
  static __device__ __forceinline__ void begin(const double* y0, const double* p, double* s) {
#pragma unroll
    for (int i = 0; i < D; ++i) { s[i] = y0[i]; s[D + i] = 0.0; }
    F::rhs(s, p, s + 2 * D);
  }
  static __device__ __forceinline__ bool attempt(const RecordArgs& a, long long j, const double* p,
                                                 const float* pf, double t1, long long rstride,
                                                 FwdCounters& c, const double* s, double* o) {
    return mixed_attempt<F>(a, j, p, pf, t1, true, true, rstride, c, s, s + D, s + 2 * D, o, o + D,
                            o + 2 * D);
  }
};

template <class F>
struct CompactRos23 {
  static constexpr int D = F::D, kState = D, QK = 6;
  static __device__ __forceinline__ void begin(const double* y0, const double*, double* s) {
#pragma unroll
    for (int i = 0; i < D; ++i) s[i] = y0[i];
  }
  static __device__ __forceinline__ bool attempt(const RecordArgs& a, long long j, const double* p,
                                                 const float*, double t1, long long rstride,
                                                 FwdCounters& c, const double* s, double* o) {
    return ros23_attempt<F>(a, j, p, t1, true, true, rstride, c, s, o);
  }
};

// Entry e of a list of capacity `cap` keeps word w at list[w * cap + e]: the state, t, dt, and
// (trajectory, attempts, accepted, rejected) in two words.
template <class M>
GS_HD int compact_words() { return M::kState + 4; }

// Entries that pass `pass` can leave behind at most: fewer than kKeep of each 32.
GS_HD long long compact_left(long long n, int pass) {
  for (int i = 0; i <= pass; ++i) n = (n + 31) / 32 * (kKeep - 1);
  return n;
}

struct CompactLists {
  const double* in;  // null: a fresh pass over all trajectories
  const int* in_count;
  double* out;       // null: the last pass
  int* out_count;
  long long in_cap, out_cap;
};

template <class F, class M, int kMinB>
__global__ void __launch_bounds__(128, kMinB) record_compact_kernel(const RecordArgs a,
                                                                    const CompactLists l) {
  constexpr int D = F::D, P = F::P, S = M::kState;
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  long long j = t;
  double sa[S], sb[S], p[P];
  float pf[P];
  FwdCounters c;
  if (l.in) {
    const long long count = *l.in_count;
    if (t >= (count < l.in_cap ? count : l.in_cap)) return;
    const double* e = l.in + t;
#pragma unroll
    for (int i = 0; i < S; ++i) sa[i] = e[i * l.in_cap];
    c.t = e[S * l.in_cap];
    c.dt = e[(S + 1) * l.in_cap];
    const long long w0 = __double_as_longlong(e[(S + 2) * l.in_cap]);
    const long long w1 = __double_as_longlong(e[(S + 3) * l.in_cap]);
    j = w0 & 0xffffffffll;
    c.it = (int)(w0 >> 32);
    c.acc = (int)(w1 & 0xffffffffll);
    c.rej = (int)(w1 >> 32);
  } else if (t >= a.n) {
    return;
  }
#pragma unroll
  for (int i = 0; i < P; ++i) { p[i] = a.p[j * P + i]; pf[i] = (float)p[i]; }
  const double t1 = a.t1v ? a.t1v[j] : a.t1;
  const long long rstride = 4 * a.n;
  if (l.in) {
    c.ck_slot = c.acc / a.ck_every;
    c.ck_cnt = c.acc - c.ck_slot * a.ck_every;
    c.rp = a.rec + ((size_t)(c.acc >> 2) * (size_t)a.n + (size_t)j) * 4u;
  } else {
    M::begin(a.y0 + j * D, p, sa);
    c.t = a.t0;
    c.dt = a.dt0 > 0.0 ? a.dt0 : (t1 - a.t0) / 100.0;
    c.it = c.acc = c.rej = c.ck_cnt = c.ck_slot = 0;
    c.rp = a.rec + j * 4;
    store_ckpt<D>(a.ckpt, a.n, j, 0, sa, c.t);
  }
  c.st = 0;
  int keep = l.out ? kKeep : 0;
  bool in_b = false;  // where the state is when the loop stops
  for (;;) {
    if (!M::attempt(a, j, p, pf, t1, rstride, c, sa, sb)) break;
    if (!M::attempt(a, j, p, pf, t1, rstride, c, sb, sa)) {
      in_b = true;
      break;
    }
    if (__popc(__activemask()) < keep) {
      const int pos = atomicAdd(l.out_count, 1);
      if (pos < l.out_cap) {
        double* e = l.out + pos;
#pragma unroll
        for (int i = 0; i < S; ++i) e[i * l.out_cap] = sa[i];
        e[S * l.out_cap] = c.t;
        e[(S + 1) * l.out_cap] = c.dt;
        e[(S + 2) * l.out_cap] = __longlong_as_double(((long long)c.it << 32) | j);
        e[(S + 3) * l.out_cap] = __longlong_as_double(((long long)c.rej << 32) | (long long)c.acc);
        return;
      }
      keep = 0;  // (a full list: to the end here)
    }
  }
  if (c.st == 0 && !(c.t >= t1)) c.st = 1;
  for (int s = c.acc; (s & 3) != 0; ++s) c.rp[s & 3] = 0.0;  // zero-pad the last sector
#pragma unroll
  for (int i = 0; i < D; ++i) a.yf[j * D + i] = in_b ? sb[i] : sa[i];
  a.n_acc[j] = c.acc;
  a.n_rej[j] = c.rej;
  a.status[j] = c.st;
}

}  // namespace gs

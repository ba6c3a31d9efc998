// O(N) Hermite-4 kernels (HBM-bound) and the FP64 energy diagnostic.
//
// Device state is SoA float64 with a padded row stride `ld` (a multiple of
// 256): X = [3][ld] positions, V = [3][ld] velocities, M = [ld] masses,
// D = [6][ld] current acc (0..2) and jerk (3..5).  Padding rows hold zero
// mass at the origin and are never integrated.
//
// Reference formulas (restated, src/nbody.cpp):
//   prediction      152-163  x += v dt + a dt^2/2 + j dt^3/6;  v += a dt + j dt^2/2
//   snapandcrackle  165-179  a2 = 2/dt^2 [-3(a - a1) - (2j + j1) dt]
//                            a3 = 6/dt^3 [ 2(a - a1) + (j + j1) dt]
//   correction      181-196  x += a2 dt^4/24 + a3 dt^5/120;  v += a2 dt^3/6 + a3 dt^4/24
//   updatedt        198-222  min_i sqrt(eta (|a||a2| + |j|^2) / (|j||a3| + |a2|^2)),
//                            with the pre-step a, j
//   initialdt       131-150  min_i eta0 |a| / |j|
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <utility>

#include "pair.cuh"
#include "symplan.h"

namespace nbody {

// Step control block in device memory; updated by the last CTA of the
// corrector so that a captured step graph needs no host round trip.
struct StepCtl {
  double dt;                       // shared step in use
  double t;                        // model time
  double dt_crit;                  // last Aarseth / initial criterion
  unsigned long long crit_bits;    // atomicMin accumulator (+inf when idle)
  unsigned int blocks_done;        // last-block detection counter
  int adaptive;                    // 1: adopt dt_crit as the next dt
  long long steps;                 // completed steps
};

// Launches a kernel that begins with grid_wait right behind the kernel before
// it on the stream: its launch overlaps that kernel's tail (three small
// kernels 7.4 us instead of 12.5).
template <class... P, class... A>
cudaError_t launch_chained(void (*k)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                           A&&... args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = grid;
  c.blockDim = block;
  c.dynamicSmemBytes = smem;
  c.stream = st;
  c.attrs = &at;
  c.numAttrs = 1;
  return cudaLaunchKernelEx(&c, k, std::forward<A>(args)...);
}

constexpr unsigned long long kPosInfBits = 0x7FF0000000000000ull;

// Deterministic block reductions for a fixed blockDim (multiple of 32, <= 1024).
__device__ __forceinline__ double block_sum(double v, double* sh) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) sh[w] = v;
  __syncthreads();
  double r = 0.0;
  if (threadIdx.x == 0)
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) r += sh[k];
  __syncthreads();
  return r;  // valid in thread 0
}

__device__ __forceinline__ double block_min(double v, double* sh) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmin(v, __shfl_xor_sync(0xffffffffu, v, o));
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) sh[w] = v;
  __syncthreads();
  double r = __longlong_as_double(static_cast<long long>(kPosInfBits));
  if (threadIdx.x == 0)
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) r = fmin(r, sh[k]);
  __syncthreads();
  return r;  // valid in thread 0
}

// Folds this CTA's criterion into ctl->crit_bits; the last CTA to finish
// publishes it and, for a step, advances t / steps (and dt when adaptive).
__device__ __forceinline__ void finish_criterion(StepCtl* ctl, double local, bool is_step,
                                                 double* sh) {
  __shared__ bool last;
  const double bmin = block_min(local, sh);
  if (threadIdx.x == 0) {
    // positive doubles order like their bit patterns; NaN (bits above +inf) never wins
    if (bmin >= 0.0) atomicMin(&ctl->crit_bits, static_cast<unsigned long long>(__double_as_longlong(bmin)));
    __threadfence();
    const unsigned prev = atomicAdd(&ctl->blocks_done, 1u);
    last = (prev == gridDim.x - 1);
  }
  __syncthreads();
  if (last && threadIdx.x == 0) {
    __threadfence();
    const unsigned long long bits = atomicExch(&ctl->crit_bits, kPosInfBits);
    const double crit = __longlong_as_double(static_cast<long long>(bits));
    ctl->dt_crit = crit;
    if (is_step) {
      ctl->t += ctl->dt;
      ctl->steps += 1;
    }
    if (ctl->adaptive && bits < kPosInfBits) ctl->dt = crit;
    ctl->blocks_done = 0;
  }
}

__device__ __forceinline__ void split_hilo(double x, float& hi, float& lo) {
  hi = __double2float_rn(x);
  lo = __double2float_rn(x - static_cast<double>(hi));
}

__device__ __forceinline__ JBody32 make_jb32(double x, double y, double z, double m, double vx,
                                             double vy, double vz) {
  JBody32 b;
  split_hilo(x, b.xh, b.xl);
  split_hilo(y, b.yh, b.yl);
  split_hilo(z, b.zh, b.zl);
  b.m = __double2float_rn(m);
  b.vx = __double2float_rn(vx);
  b.vy = __double2float_rn(vy);
  b.vz = __double2float_rn(vz);
  b.pad0 = b.pad1 = 0.f;
  return b;
}

__device__ __forceinline__ JBodyX2 make_jbx2(double x, double y, double z, double m, double vx,
                                             double vy, double vz) {
  const JBody32 b = make_jb32(x, y, z, m, vx, vy, vz);
  JBodyX2 d;
  d.xh = make_float2(b.xh, b.xh); d.yh = make_float2(b.yh, b.yh); d.zh = make_float2(b.zh, b.zh);
  d.m = make_float2(b.m, b.m);
  d.xl = make_float2(b.xl, b.xl); d.yl = make_float2(b.yl, b.yl); d.zl = make_float2(b.zl, b.zl);
  d.vx = make_float2(b.vx, b.vx); d.vy = make_float2(b.vy, b.vy); d.vz = make_float2(b.vz, b.vz);
  d.pad0 = d.pad1 = make_float2(0.f, 0.f);
  return d;
}

// j-record formats of the pair kernels.
enum RecordFormat { kRecF64 = 0, kRecF32 = 1, kRecX2 = 2, kRecRel = 3, kRecSym = 4 };

// Seven SoA input arrays (caller's or the engine's own).
struct SoA7 {
  const double *x, *y, *z, *m, *vx, *vy, *vz;
};
// Six SoA output arrays.
struct SoA6 {
  double *ax, *ay, *az, *jx, *jy, *jz;
};

// Writes j-records for rows [0, ld): rows < n from `in`, the rest as
// zero-mass bodies at rest at the origin (they contribute exactly zero).
static __global__ void pack_kernel(int n, int ld, SoA7 in, JBody64* __restrict__ jb64,
                            JBody32* __restrict__ jb32, JBodyX2* __restrict__ jbx2 = nullptr) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= ld) return;
  double x = 0, y = 0, z = 0, m = 0, vx = 0, vy = 0, vz = 0;
  if (i < n) {
    x = in.x[i]; y = in.y[i]; z = in.z[i]; m = in.m[i];
    vx = in.vx[i]; vy = in.vy[i]; vz = in.vz[i];
  }
  if (jb64) store_jb64(jb64, i, x, y, z, m, vx, vy, vz);
  if (jb32) jb32[i] = make_jb32(x, y, z, m, vx, vy, vz);
  if (jbx2) jbx2[i] = make_jbx2(x, y, z, m, vx, vy, vz);
}

// One component's predicted position and velocity.
__device__ __forceinline__ void predict_component(double dt, double x, double v, double a, double j,
                                                  double& p, double& u) {
  const double h2 = 0.5 * dt * dt;
  const double h3 = dt * dt * dt * (1.0 / 6.0);
  p = x + (v * dt + (a * h2 + j * h3));
  u = v + (a * dt + j * h2);
}

// Predicted position p and velocity u of row i, written back to X, V and, if
// not null, to XP ([6][ld]).
__device__ __forceinline__ void predict_body(double dt, int ld, int i, double* __restrict__ X,
                                             double* __restrict__ V, const double* __restrict__ D,
                                             double p[3], double u[3],
                                             double* __restrict__ XP = nullptr) {
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    predict_component(dt, X[c * ld + i], V[c * ld + i], D[c * ld + i], D[(3 + c) * ld + i], p[c], u[c]);
    X[c * ld + i] = p[c];
    V[c * ld + i] = u[c];
    if (XP) {
      XP[c * ld + i] = p[c];
      XP[(3 + c) * ld + i] = u[c];
    }
  }
}

// Predictor: in place on X, V (rows < n) and writes the j-records of the
// predicted state (jb64 or jb32, whichever is non-null).
static __global__ void predict_kernel(int n, int ld, const StepCtl* __restrict__ ctl, double* __restrict__ X,
                               double* __restrict__ V, const double* __restrict__ M,
                               const double* __restrict__ D, JBody64* __restrict__ jb64,
                               JBody32* __restrict__ jb32, JBodyX2* __restrict__ jbx2,
                               double* __restrict__ XP = nullptr) {
  grid_wait();
  grid_release();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double p[3], u[3];
  predict_body(ctl->dt, ld, i, X, V, D, p, u, XP);
  const double m = M[i];
  if (jb64) store_jb64(jb64, i, p[0], p[1], p[2], m, u[0], u[1], u[2]);
  if (jb32) jb32[i] = make_jb32(p[0], p[1], p[2], m, u[0], u[1], u[2]);
  if (jbx2) jbx2[i] = make_jbx2(p[0], p[1], p[2], m, u[0], u[1], u[2]);
}

// sum[c] = sum over slots s = 0, 1, ..., S-1 (in that order) of
// P[s * step][c][i], for the F fields at once: one pass over the splits with
// several loads in flight, so a small system (few CTAs) is not bound by
// one load latency per split.
template <int F = 6>
__device__ __forceinline__ void split_sums(const double* __restrict__ P, int ld, int S, int i,
                                           double sum[F], int step = 1) {
#pragma unroll
  for (int c = 0; c < F; ++c) sum[c] = 0.0;
#pragma unroll 4
  for (int s = 0; s < S; ++s) {
    const double* p = P + static_cast<size_t>(s) * step * F * ld + i;
#pragma unroll
    for (int c = 0; c < F; ++c) sum[c] += p[static_cast<size_t>(c) * ld];
  }
}

// Threads of the kernels that sum slots: kSumThreads per CTA, as kSumThreads /
// GR rows times GR groups.  Group g adds the slots g, g + GR, ... of its row,
// and the groups' sums are added in group order through shared memory, so a
// result's rounding depends on GR but not on timing.  A small system has few
// rows and, with the symmetric kernels, dozens of slots: with one thread per
// row its sums are a chain of loads on a handful of SMs.
constexpr int kSumThreads = 256;
template <int GR>
constexpr int kSumRows = kSumThreads / GR;

// The F sums of row i, valid in the threads of group 0 (threadIdx.x <
// kSumRows<GR>); sh holds F * kSumThreads doubles when GR > 1.
template <int GR, int F = 6>
__device__ __forceinline__ void slot_sums(const double* __restrict__ P, int ld, int S, int i,
                                          double sum[F], double* sh) {
  constexpr int R = kSumRows<GR>;
  const int g = threadIdx.x / R, r = threadIdx.x % R;
  split_sums<F>(P + static_cast<size_t>(g) * F * ld, ld, (S - g + GR - 1) / GR, i, sum, GR);
  if (GR > 1) {
#pragma unroll
    for (int c = 0; c < F; ++c) sh[(g * F + c) * R + r] = sum[c];
    __syncthreads();
    if (g == 0)
#pragma unroll
      for (int q = 1; q < GR; ++q)
#pragma unroll
        for (int c = 0; c < F; ++c) sum[c] += sh[(q * F + c) * R + r];
  }
}

// The corrector of row i (the calling thread's): snap/crackle from the pre-step
// d = (a, j) and the new sums, corrected x, v in place; returns the Aarseth
// criterion.
__device__ __forceinline__ double correct_body(double dt, double eta, const double d[6],
                                               const double sum[6], double x[3], double v[3]) {
  const double idt2 = 1.0 / (dt * dt);
  const double idt3 = idt2 / dt;
  const double dt3 = dt * dt * dt, dt4 = dt3 * dt, dt5 = dt4 * dt;
  double A2 = 0, J2 = 0, S2 = 0, C2 = 0;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const double a1 = sum[c], j1 = sum[3 + c];
    const double a = d[c], j = d[3 + c];
    const double da = a - a1;
    const double a2 = 2.0 * idt2 * (-3.0 * da - (2.0 * j + j1) * dt);
    const double a3 = 6.0 * idt3 * (2.0 * da + (j + j1) * dt);
    x[c] += a2 * dt4 * (1.0 / 24.0) + a3 * dt5 * (1.0 / 120.0);
    v[c] += a2 * dt3 * (1.0 / 6.0) + a3 * dt4 * (1.0 / 24.0);
    A2 += a * a; J2 += j * j; S2 += a2 * a2; C2 += a3 * a3;
  }
  const double num = sqrt(A2) * sqrt(S2) + J2;
  const double den = sqrt(J2) * sqrt(C2) + S2;
  return sqrt(eta * num / den);
}

// Corrector fused with the split-j reduction and the Aarseth criterion:
// a1/j1 = sum over the row's slots of P; snap/crackle; correct X, V; D <- a1/j1.
// PREDICT (fixed step only: an adaptive one is known when every row is done):
// the next step's predictor on top, so X, V become its predicted state and jb64
// its records; M: masses.
template <int GR, bool PREDICT = false>
static __global__ void __launch_bounds__(kSumThreads)
    correct_kernel(int n, int ld, RowSlots slots, const double* __restrict__ P,
                   double* __restrict__ X, double* __restrict__ V, double* __restrict__ D,
                   StepCtl* __restrict__ ctl, double eta, const double* __restrict__ M = nullptr,
                   JBody64* __restrict__ jb64 = nullptr) {
  __shared__ double sh[GR > 1 ? 6 * kSumThreads : 32];
  grid_wait();
  grid_release();
  const int i = blockIdx.x * kSumRows<GR> + threadIdx.x % kSumRows<GR>;
  double crit = __longlong_as_double(static_cast<long long>(kPosInfBits));
  const bool mine = i < n && threadIdx.x < kSumRows<GR>;
  double x[3], v[3], d[6];
  if (mine)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      x[c] = X[c * ld + i]; v[c] = V[c * ld + i];
      d[c] = D[c * ld + i]; d[3 + c] = D[(3 + c) * ld + i];
    }
  double sum[6];
  slot_sums<GR>(P, ld, i < n ? slots.count(i) : 0, i, sum, sh);
  if (mine) {
    const double dt = ctl->dt;
    crit = correct_body(dt, eta, d, sum, x, v);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      if (PREDICT) predict_component(dt, x[c], v[c], sum[c], sum[3 + c], x[c], v[c]);
      X[c * ld + i] = x[c];
      V[c * ld + i] = v[c];
      D[c * ld + i] = sum[c];
      D[(3 + c) * ld + i] = sum[3 + c];
    }
    if (PREDICT) store_jb64(jb64, i, x[0], x[1], x[2], M[i], v[0], v[1], v[2]);
  }
  if (GR > 1) __syncthreads();  // sh is reused
  finish_criterion(ctl, crit, true, sh);
}

// out[c][i] = sum over the row's slots of P for rows [i_begin, i_end).
// With a status word (callers that cannot read it back before using the
// outputs), a non-zero word - a pair kernel gave up a bounded wait - makes
// every output NaN instead.  With an index map, row i is written to
// out[c][index[i]] (partials kept in Hilbert order, outputs in the caller's
// body order).
template <int GR>
static __global__ void __launch_bounds__(kSumThreads)
    reduce_splits_kernel(int i_begin, int i_end, int ld, RowSlots slots,
                         const double* __restrict__ P, SoA6 out,
                         const int* __restrict__ status = nullptr,
                         const int* __restrict__ index = nullptr) {
  __shared__ double sh[GR > 1 ? 6 * kSumThreads : 1];
  const int i = i_begin + blockIdx.x * kSumRows<GR> + threadIdx.x % kSumRows<GR>;
  double sum[6];
  slot_sums<GR>(P, ld, i < i_end ? slots.count(i) : 0, i, sum, sh);
  if (i >= i_end || threadIdx.x >= kSumRows<GR>) return;
  double* dst[6] = {out.ax, out.ay, out.az, out.jx, out.jy, out.jz};
  const int o = index ? index[i] : i;
  const bool bad = status && *status != 0;
#pragma unroll
  for (int c = 0; c < 6; ++c)
    dst[c][o] = bad ? __longlong_as_double(0x7FF8000000000000ll) : sum[c];
}

// One field of reduce_splits_kernel: out[index ? index[i] : i] = sum over
// the row's slots of P[(s*6 + c)*ld + i], for the field c whose [ld] block of
// slot 0 is Pc.  Lets a caller copy each finished field to the host while the
// next one reduces.
template <int GR>
static __global__ void __launch_bounds__(kSumThreads)
    reduce_split_field_kernel(int i_begin, int i_end, int ld, RowSlots slots,
                              const double* __restrict__ Pc, double* __restrict__ out,
                              const int* __restrict__ index = nullptr) {
  constexpr int R = kSumRows<GR>;
  __shared__ double sh[kSumThreads];
  const int g = threadIdx.x / R, r = threadIdx.x % R;
  const int i = i_begin + blockIdx.x * R + r;
  const int S = i < i_end ? slots.count(i) : 0;
  double sum = 0.0;
#pragma unroll 8
  for (int s = g; s < S; s += GR) sum += Pc[static_cast<size_t>(s) * 6 * ld + i];
  if (GR > 1) {
    sh[threadIdx.x] = sum;
    __syncthreads();
    if (g == 0)
#pragma unroll
      for (int q = 1; q < GR; ++q) sum += sh[q * R + r];
  }
  if (g == 0 && i < i_end) out[index ? index[i] : i] = sum;
}

// Groups per row: eight from kSumGroupSlots slots, one below, where most
// groups would have nothing to add.  Corrector with eight groups against one,
// cold caches, N = 4096: 9.7 us over 44 slots against 18.6 over 32; a step at N =
// 1024 39.4 against 42.4 us.  At N = 65536 the partials' bandwidth bounds both:
// the same within 0.2 % of a step over 80 slots; over the 116 (mixed) and 106
// (FP64) of the automatic splits eight groups take 96 and 92 us, 3.9 TB/s.
constexpr int kSumGroupSlots = 8;
inline bool sum_in_groups(const RowSlots& s) { return s.S + s.nb / 2 >= kSumGroupSlots; }

inline void launch_correct(cudaStream_t st, int n, int ld, RowSlots slots, const double* P,
                           double* X, double* V, double* D, StepCtl* ctl, double eta,
                           bool chained = false) {
  if (sum_in_groups(slots) && chained)
    launch_chained(correct_kernel<8>, (n + kSumRows<8> - 1) / kSumRows<8>, kSumThreads, 0, st, n, ld,
                   slots, P, X, V, D, ctl, eta, static_cast<const double*>(nullptr), static_cast<JBody64*>(nullptr));
  else if (sum_in_groups(slots))
    correct_kernel<8><<<(n + kSumRows<8> - 1) / kSumRows<8>, kSumThreads, 0, st>>>(
        n, ld, slots, P, X, V, D, ctl, eta);
  else
    correct_kernel<1><<<(n + kSumRows<1> - 1) / kSumRows<1>, kSumThreads, 0, st>>>(
        n, ld, slots, P, X, V, D, ctl, eta);
}
inline void launch_reduce(cudaStream_t st, int i_begin, int i_end, int ld, RowSlots slots,
                          const double* P, SoA6 out, const int* status = nullptr,
                          const int* index = nullptr) {
  const int rows = i_end - i_begin;
  if (sum_in_groups(slots))
    reduce_splits_kernel<8><<<(rows + kSumRows<8> - 1) / kSumRows<8>, kSumThreads, 0, st>>>(
        i_begin, i_end, ld, slots, P, out, status, index);
  else
    reduce_splits_kernel<1><<<(rows + kSumRows<1> - 1) / kSumRows<1>, kSumThreads, 0, st>>>(
        i_begin, i_end, ld, slots, P, out, status, index);
}
inline void launch_reduce_field(cudaStream_t st, int i_begin, int i_end, int ld, RowSlots slots,
                                const double* Pc, double* out, const int* index) {
  const int rows = i_end - i_begin;
  if (sum_in_groups(slots))
    reduce_split_field_kernel<8><<<(rows + kSumRows<8> - 1) / kSumRows<8>, kSumThreads, 0, st>>>(
        i_begin, i_end, ld, slots, Pc, out, index);
  else
    reduce_split_field_kernel<1><<<(rows + kSumRows<1> - 1) / kSumRows<1>, kSumThreads, 0, st>>>(
        i_begin, i_end, ld, slots, Pc, out, index);
}

// Initial step criterion min_i eta0 |a| / |j| (published via ctl).
static __global__ void initialdt_kernel(int n, int ld, const double* __restrict__ D, StepCtl* ctl,
                                 double eta0) {
  __shared__ double sh[32];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  double crit = __longlong_as_double(static_cast<long long>(kPosInfBits));
  if (i < n) {
    const double a0 = D[i], a1 = D[ld + i], a2 = D[2 * ld + i];
    const double j0 = D[3 * ld + i], j1 = D[4 * ld + i], j2 = D[5 * ld + i];
    crit = eta0 * sqrt(a0 * a0 + a1 * a1 + a2 * a2) / sqrt(j0 * j0 + j1 * j1 + j2 * j2);
  }
  finish_criterion(ctl, crit, false, sh);
}

// FP64 records of the energy diagnostic (rows [0, ld), padding zero) and per-CTA
// partials of 0.5 m v^2.
static __global__ void energy_pack_kernel(int n, int ld, SoA7 in, JBody64* __restrict__ jb,
                                          double* __restrict__ partial) {
  __shared__ double sh[32];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  double e = 0.0;
  if (i < n) {
    const double m = in.m[i], u = in.vx[i], v = in.vy[i], w = in.vz[i];
    e = 0.5 * m * (u * u + v * v + w * w);
    store_jb64(jb, i, in.x[i], in.y[i], in.z[i], m, u, v, w);
  } else if (i < ld) {
    store_jb64(jb, i, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0);
  }
  const double b = block_sum(e, sh);
  if (threadIdx.x == 0) partial[blockIdx.x] = b;
}

// out[b] = the sum of count[b] partials, in a fixed order (CTA b of two).
static __global__ void sum_partials_kernel(int count0, const double* __restrict__ partial0, int count1,
                                           const double* __restrict__ partial1,
                                           double* __restrict__ out) {
  __shared__ double sh[32];
  const int count = blockIdx.x ? count1 : count0;
  const double* p = blockIdx.x ? partial1 : partial0;
  double v = 0.0;
  for (int k = threadIdx.x; k < count; k += blockDim.x) v += p[k];
  const double b = block_sum(v, sh);
  if (threadIdx.x == 0) out[blockIdx.x] = b;
}

}  // namespace nbody

// Reverse-mode gradients of a fixed-dt Hermite-4 trajectory.
//
// Step map (shared step h), per body, with the corrector written out:
//   predict   xp = x0 + h v0 + h^2/2 a0 + h^3/6 j0,   vp = v0 + h a0 + h^2/2 j0
//   evaluate  (a1, j1) = F(xp, vp, m)                      (the pair acc + jerk)
//   correct   x1 = xp - 0.15 h^2 (a0 - a1) - h^3 (7/60 j0 + 1/30 j1)
//             v1 = vp - 0.5  h   (a0 - a1) - h^2 (5/12 j0 + 1/12 j1)
// (the last two lines are a2 h^4/24 + a3 h^5/120 and a2 h^3/6 + a3 h^4/24
// with the reference's snap/crackle, src/nbody.cpp:165-196, expanded).  The
// state carried between steps is (x, v, a, j); the initial (a0, j0) is
// F(x_init, v_init, m).
//
// Backward: adjoints (xb, vb, ab, jb) of a step's outputs give those of its
// inputs through
//   pre   ab1 = 0.15 h^2 xb1 + 0.5 h vb1 + ab_out,  jb1 = -(h^3/30) xb1 - (h^2/12) vb1 + jb_out
//         ab0 = -0.15 h^2 xb1 - 0.5 h vb1,          jb0 = -(7 h^3/60) xb1 - (5 h^2/12) vb1
//   VJP   (xbp, vbp, mb) += F^T (ab1, jb1) at (xp, vp, m);  xbp, vbp start at xb1, vb1
//   post  xb0 = xbp, vb0 = h xbp + vbp,  ab0 += h^2/2 xbp + h vbp,  jb0 += h^3/6 xbp + h^2/2 vbp
// The forward keeps the state every `checkpoint_every` steps; the backward
// restores each segment's checkpoint, recomputes its steps keeping the
// predicted (xp, vp), and runs the reverse steps.  The pair VJP is FP64 for
// both precisions (for a mixed-precision forward it is the FP64 adjoint of
// the same trajectory).
//
// Pair VJP (no atomics).  For an unordered pair (k, p) with r = x_p - x_k,
// u = v_p - v_k, s = r^2 + eps2, y2 = 1/s, q = s^(-3/2), w = r.u, c = -3 w y2
// and the adjoints (a, b) = (ab, jb) of acc and jerk, both bodies' terms are
//   T = q (m_p G_k - m_k G_p),  G_i = a_i.r + b_i.u + c B_i,  B_i = b_i.r
// (body p sees -r and -u).  With A = m_p a_k - m_k a_p, J = m_p b_k - m_k b_p,
// B = m_p B_k - m_k B_p and G = m_p G_k - m_k G_p:
//   dT/dr = q [A + c J - 3 y2 B u - 3 y2 (G + 2/3 c B) r],  dT/du = q (J - 3 y2 B r),
//   dT/dm_p = q G_k,  dT/dm_k = -q G_p.
// x_p collects +dT/dr and x_k -dT/dr, likewise v.  The symmetric schedule
// (sympair.cuh) meets every pair once: 87 FP64 operations for both bodies.
#include <cuda_runtime.h>

#include <algorithm>
#include <memory>
#include <vector>

#include "../../include/nbody_cuda.h"
#include "devptr.h"
#include "errors.h"
#include "hermite.cuh"
#include "pair.cuh"
#include "sympair.cuh"
#include "trace.h"

using namespace nbody;

namespace {

constexpr int kPad = 256;
constexpr int kBlock = 256;
constexpr int kPredictBlock = 64;  // a few thousand rows reach more SMs

// j-record of the pair VJP, in groups of 32 bodies, each seven rows of 32
// 16-byte chunks: (x, y) (z, m) (vx, vy) (vz, ax) (ay, az) (bx, by) (bz, -)
// with (a, b) the acc/jerk adjoints.  JAdj is one body's share of a group.
constexpr int kAdjChunks = 7;
struct __align__(16) JAdj {
  double raw[2 * kAdjChunks];
};
constexpr int kVjpTile = 32;

__device__ __forceinline__ double2* jadj_at(JAdj* jb, int i) {
  return reinterpret_cast<double2*>(jb + (i & ~31)) + (i & 31);
}

// One body's values.
struct VjpBody {
  double x, y, z, m, u, v, w, ax, ay, az, bx, by, bz;
  __device__ __forceinline__ void load(const double2* p) {
    const double2 p0 = p[0], p1 = p[32], p2 = p[64], p3 = p[96], p4 = p[128], p5 = p[160], p6 = p[192];
    x = p0.x; y = p0.y; z = p1.x; m = p1.y; u = p2.x; v = p2.y; w = p3.x;
    ax = p3.y; ay = p4.x; az = p4.y; bx = p5.x; by = p5.y; bz = p6.x;
  }
};

// The pair (k, p): ai and (SYM) bj collect q dT/dr, q dT/du and the masses'
// terms; the row's sums change sign when they are stored.  skip: the self
// pair, whose terms are finite and taken out by q = 0.
template <bool SYM>
__device__ __forceinline__ void vjp_pair(const VjpBody& k, const VjpBody& p, double eps2, bool skip,
                                         double* ai, double* bj) {
  const double r0 = p.x - k.x, r1 = p.y - k.y, r2 = p.z - k.z;
  const double u0 = p.u - k.u, u1 = p.v - k.v, u2 = p.w - k.w;
  const double s = fma(r0, r0, fma(r1, r1, fma(r2, r2, eps2)));
  const double wr = fma(r0, u0, fma(r1, u1, r2 * u2));
  const double y = rsqrt_f64(s);
  const double y2 = y * y;
  const double q = !SYM && skip ? 0.0 : y * y2;
  const double t = -3.0 * y2, c = wr * t;
  const double Bk = fma(k.bx, r0, fma(k.by, r1, k.bz * r2));
  const double Bp = fma(p.bx, r0, fma(p.by, r1, p.bz * r2));
  const double Gk = fma(c, Bk, fma(k.ax, r0, fma(k.ay, r1, fma(k.az, r2, fma(k.bx, u0, fma(k.by, u1, k.bz * u2))))));
  const double Gp = fma(c, Bp, fma(p.ax, r0, fma(p.ay, r1, fma(p.az, r2, fma(p.bx, u0, fma(p.by, u1, p.bz * u2))))));
  const double B = fma(p.m, Bk, -(k.m * Bp)), G = fma(p.m, Gk, -(k.m * Gp));
  const double J0 = fma(p.m, k.bx, -(k.m * p.bx)), J1 = fma(p.m, k.by, -(k.m * p.by)),
               J2 = fma(p.m, k.bz, -(k.m * p.bz));
  const double A0 = fma(c, J0, fma(p.m, k.ax, -(k.m * p.ax))), A1 = fma(c, J1, fma(p.m, k.ay, -(k.m * p.ay))),
               A2 = fma(c, J2, fma(p.m, k.az, -(k.m * p.az)));
  const double e = t * B, kr = t * fma(c * (2.0 / 3.0), B, G);
  const double d0 = fma(kr, r0, fma(e, u0, A0)), d1 = fma(kr, r1, fma(e, u1, A1)), d2 = fma(kr, r2, fma(e, u2, A2));
  const double g0 = fma(e, r0, J0), g1 = fma(e, r1, J1), g2 = fma(e, r2, J2);
  ai[0] = fma(q, d0, ai[0]); ai[1] = fma(q, d1, ai[1]); ai[2] = fma(q, d2, ai[2]);
  ai[3] = fma(q, g0, ai[3]); ai[4] = fma(q, g1, ai[4]); ai[5] = fma(q, g2, ai[5]);
  ai[6] = fma(q, Gp, ai[6]);
  if (SYM) {
    bj[0] = fma(q, d0, bj[0]); bj[1] = fma(q, d1, bj[1]); bj[2] = fma(q, d2, bj[2]);
    bj[3] = fma(q, g0, bj[3]); bj[4] = fma(q, g1, bj[4]); bj[5] = fma(q, g2, bj[5]);
    bj[6] = fma(q, Gk, bj[6]);
  }
}

// Slots [slot][7][ld]: d(xbar) (3), d(vbar) (3), d(mbar).  Bound by the FP64
// pipe; two rows per lane put the 14 shuffles and seven 16-byte shared loads
// of a step (42 cycles of the shared pipe) under 2 x 87 FP64 instructions (87
// cycles).  One row or three CTAs per SM time the same within 3 %.  Whole call
// against the one-sided gather form: N = 4096 224 vs 297 us, 8192 399 vs 639,
// 20000 1543 vs 3121.
template <int IPT, int W>
constexpr size_t vjp_smem() {
  return 2 * kVjpTile * sizeof(JAdj) + 2 * 7 * W * 32 * sizeof(double);
}
template <int IPT, int W, int UNR, int MINB>
__global__ void __launch_bounds__(32 * W, MINB) vjp_sym_kernel(JAdj* __restrict__ jb, SymArgs a) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ uint64_t full[2];
  constexpr int kRows = 32 * IPT * W;
  static_assert(kRows % kVjpTile == 0, "blocks are whole tiles");
  TilePipe<JAdj, kVjpTile> pipe;
  pipe.init(reinterpret_cast<JAdj*>(smem_raw), full);
  double* red = reinterpret_cast<double*>(smem_raw + 2 * kVjpTile * sizeof(JAdj));  // [2][7][W][32]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, next = (lane + 1) & 31;
  const SymRun run(a, a.subs * (kRows / kVjpTile));
  const double eps2 = a.eps2;
  int half = 0;
  grid_wait();
  for (int g = 0; g < a.subs; ++g) {
    const int row0 = (run.I * a.subs + g) * kRows + warp * 32 * IPT;
    if ((run.I * a.subs + g) * kRows >= a.n) break;  // a short last block
    VjpBody me[IPT];
    double acc[IPT][7];
#pragma unroll
    for (int k = 0; k < IPT; ++k) {
      const int r = row0 + 32 * k + lane;
      // rows in [n, ld) are zero records; rows past ld have none (zero mass and
      // adjoints add nothing, and they are not stored)
      me[k] = VjpBody{};
      if (r < a.ld) me[k].load(jadj_at(jb, r));
#pragma unroll
      for (int c = 0; c < 7; ++c) acc[k][c] = 0.0;
    }
    int t = 0;
    auto consume = [&](const JAdj* tile) {
      const double2* p = reinterpret_cast<const double2*>(tile);
      const int tt = run.tile(t);
      VjpBody o;
      if (run.distance(tt) == 0) {
#pragma unroll 1
        for (int k = 0; k < 32; ++k) {
          o.load(p + k);
          const int j = tt * kVjpTile + k;
#pragma unroll
          for (int r = 0; r < IPT; ++r)
            vjp_pair<false>(me[r], o, eps2, j == row0 + 32 * r + lane, acc[r], nullptr);
        }
      } else {
        double b[7] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
#pragma unroll UNR
        for (int k = 0; k < 32; ++k) {
          o.load(p + ((lane + k) & 31));
#pragma unroll
          for (int r = 0; r < IPT; ++r) vjp_pair<true>(me[r], o, eps2, false, acc[r], b);
#pragma unroll
          for (int c = 0; c < 7; ++c) b[c] = __shfl_sync(0xffffffffu, b[c], next);
        }
        double* w = red + half * 7 * W * 32 + warp * 32 + lane;
#pragma unroll
        for (int c = 0; c < 7; ++c) w[c * W * 32] = b[c];
      }
    };
    auto post = [&]() {  // the tile's sums over the W warps, into their slot
      const int tt = run.tile(t), d = run.distance(tt);
      if (d != 0) {
        const double* o = red + half * 7 * W * 32;
        double* out = a.out + static_cast<size_t>(a.S + d - 1) * 7 * a.stride +
                      static_cast<size_t>(tt) * kVjpTile;
        for (int e = threadIdx.x; e < 7 * 32; e += 32 * W) {
          const int l = e & 31, c = e >> 5;
          double v = 0.0;
#pragma unroll
          for (int w = 0; w < W; ++w) v += o[(c * W + w) * 32 + l];
          double* dst = out + static_cast<size_t>(c) * a.stride + l;
          *dst = g ? *dst + v : v;  // a later sub-block adds to this thread's own store
        }
      }
      ++t;
      half ^= 1;
    };
    if (!run.stream(pipe, jb, a.status, consume, post)) return;
    if (g + 1 == a.subs) grid_release();
    double* out = a.out + static_cast<size_t>(blockIdx.y) * 7 * a.stride;
#pragma unroll
    for (int k = 0; k < IPT; ++k) {
      const int r = row0 + 32 * k + lane;
      if (r < a.n)
#pragma unroll
        for (int c = 0; c < 7; ++c) out[static_cast<size_t>(c) * a.stride + r] = -acc[k][c];
    }
  }
}

// Everything between two pair VJPs, per row, in one pass (it was five: slot
// sums, reverse predictor, reverse corrector, adjoint and record packing, each
// a launch on a handful of SMs for systems of a few thousand bodies).  ADJ =
// [xb(3) vb(3) ab(3) jb(3)][ld], MB the mass adjoint.
//   sum   adds the finished VJP's slots to xb, vb and MB
//   post  reverse predictor: (xbp, vbp) -> (xb0, vb0), ab0/jb0 completed
//   pack  the next VJP's records at state XV ([6][ld]), with the acc/jerk adjoints
//         kPackStep  of the reverse corrector of the step whose outputs ADJ now
//                    holds (its own part of ab0/jb0 goes to ADJ's ab/jb slots)
//         kPackFrom  AB ([6][ld])
// Rows >= n pack as zero records.
enum AdjPack { kPackNone, kPackStep, kPackFrom };
__global__ void __launch_bounds__(kSumThreads)
    adj_link_kernel(int n, int ld, double h, RowSlots slots, bool sum, const double* __restrict__ P,
                    bool post, double* ADJ, double* __restrict__ MB, int pack,
                    const double* __restrict__ XV, const double* __restrict__ M, const double* AB,
                    JAdj* __restrict__ jb) {
  constexpr int GR = 8;
  __shared__ double sh[7 * kSumThreads];
  grid_wait();
  grid_release();
  const int i = blockIdx.x * kSumRows<GR> + threadIdx.x % kSumRows<GR>;
  double d[7];
  if (sum) slot_sums<GR, 7>(P, ld, i < n ? slots.count(i) : 0, i, d, sh);
  if (threadIdx.x >= kSumRows<GR> || i >= ld) return;
  const bool real = i < n;
  const double h2 = h * h, h3 = h2 * h;
  double a[3] = {0.0, 0.0, 0.0}, b[3] = {0.0, 0.0, 0.0};
  if (real) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      double xb = ADJ[c * ld + i], vb = ADJ[(3 + c) * ld + i];
      double ab = ADJ[(6 + c) * ld + i], jb_ = ADJ[(9 + c) * ld + i];
      if (sum) {
        xb += d[c];
        vb += d[3 + c];
      }
      if (post) {
        ab += 0.5 * h2 * xb + h * vb;
        jb_ += (h3 / 6.0) * xb + 0.5 * h2 * vb;
        vb = h * xb + vb;
      }
      if (pack == kPackStep) {
        a[c] = 0.15 * h2 * xb + 0.5 * h * vb + ab;
        b[c] = -(h3 / 30.0) * xb - (h2 / 12.0) * vb + jb_;
        ab = -0.15 * h2 * xb - 0.5 * h * vb;
        jb_ = -(7.0 * h3 / 60.0) * xb - (5.0 * h2 / 12.0) * vb;
      } else if (pack == kPackFrom) {
        a[c] = AB[c * ld + i];
        b[c] = AB[(3 + c) * ld + i];
      }
      ADJ[c * ld + i] = xb;
      ADJ[(3 + c) * ld + i] = vb;
      ADJ[(6 + c) * ld + i] = ab;
      ADJ[(9 + c) * ld + i] = jb_;
    }
    if (sum) MB[i] += d[6];
  }
  if (pack != kPackNone) {
    double2* o = jadj_at(jb, i);
    const double z = 0.0;
    o[0] = make_double2(real ? XV[i] : z, real ? XV[ld + i] : z);
    o[32] = make_double2(real ? XV[2 * ld + i] : z, real ? M[i] : z);
    o[64] = make_double2(real ? XV[3 * ld + i] : z, real ? XV[4 * ld + i] : z);
    o[96] = make_double2(real ? XV[5 * ld + i] : z, a[0]);
    o[128] = make_double2(a[1], a[2]);
    o[160] = make_double2(b[0], b[1]);
    o[192] = make_double2(b[2], z);
  }
}

// dst[a][i] = src[a][i] for rows i < n of g.arrays arrays (one launch instead
// of a copy per array); rows [n, ld) of `dst` become zero when pad is set.
__global__ void copy_rows_kernel(int n, int ld, GatherArgs g, bool pad) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (pad ? ld : n)) return;
#pragma unroll
  for (int a = 0; a < kMaxGather; ++a)
    if (a < g.arrays) g.dst[a][i] = i < n && g.src[a] ? g.src[a][i] : 0.0;
}

#define AD_CUDA(call)                                                                      \
  do {                                                                                     \
    cudaError_t e_ = (call);                                                               \
    if (e_ != cudaSuccess) {                                                               \
      cudaGetLastError(); /* returned here, not by the next call's check of its launches */ \
      return nbody_set_error(e_ == cudaErrorMemoryAllocation ? NBODY_ERR_OOM : NBODY_ERR_CUDA, \
                             "%s failed: %s", #call, cudaGetErrorString(e_));              \
    }                                                                                      \
  } while (0)
#define AD_TRY(expr)               \
  do {                             \
    nbody_status s_ = (expr);      \
    if (s_ != NBODY_OK) return s_; \
  } while (0)

// Symmetric kernels of the forward (two and four rows per lane, as the engine)
// and of the VJP.
constexpr int kW = 4;  // warps per CTA
const void* fwd_fp64(bool wide) {
  return wide ? reinterpret_cast<const void*>(&pair_sym_fp64_kernel<4, kW, 2, 2>)
              : reinterpret_cast<const void*>(&pair_sym_fp64_kernel<2, kW, 4, 4>);
}
const void* fwd_mixed(bool wide) {
  return wide ? reinterpret_cast<const void*>(&pair_sym_nf_kernel<4, kW, 2, 4, 2, 3>)
              : reinterpret_cast<const void*>(&pair_sym_nf_kernel<2, kW, 1, 4, 8, 4>);
}
const void* vjp_fn() { return reinterpret_cast<const void*>(&vjp_sym_kernel<2, kW, 2, 2>); }

// A symmetric kernel with its grid for one system size.
struct SymLaunch {
  const void* fn = nullptr;
  size_t smem = 0;
  int rows = 0, tj = 0, S = 1, subs = 1, nb = 1, block_rows = 1;
  double ms = 0;  // predicted
  cudaError_t plan(const void* f, size_t sm, int rows_, int tj_, int n, int sms, double rate, double tail,
                   int most_slots) {
    fn = f; smem = sm; rows = rows_; tj = tj_;
    cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(sm));
    if (e != cudaSuccess) return e;
    int occ = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, f, 32 * kW, sm);
    if (e != cudaSuccess) return e;
    const SymPlan p = sym_plan(sms, std::max(occ, 1), rows, tj, n, rate, tail, most_slots);
    S = p.S;
    ms = p.ms;
    const SymGrid g(rows, n, most_slots);
    subs = g.subs; nb = g.nb; block_rows = g.block_rows;
    return cudaSuccess;
  }
  RowSlots slots() const { return RowSlots(S, block_rows, nb); }
  size_t count() const { return S + nb / 2; }
  cudaError_t launch(const void* records, SymArgs a, cudaStream_t st) const {
    a.nb = nb; a.subs = subs; a.S = S;
    a.tiles = (a.n + tj - 1) / tj;
    void* args[] = {static_cast<void*>(&records), static_cast<void*>(&a)};
    cudaLaunchAttribute at{};  // as launch_chained
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = dim3(nb, S);
    c.blockDim = dim3(32 * kW);
    c.dynamicSmemBytes = smem;
    c.stream = st;
    c.attrs = &at;
    c.numAttrs = 1;
    return cudaLaunchKernelExC(&c, fn, args);
  }
};

}  // namespace

struct nbody_adjoint {
  nbody_adjoint_config cfg{};
  int n = 0, ld = 0, sms = 0, nseg = 0;
  double* state = nullptr;  // [13][ld]: X V M D
  double *X = nullptr, *V = nullptr, *M = nullptr, *D = nullptr;
  double* ckpt = nullptr;   // [nseg][13][ld]
  double* segxv = nullptr;  // [checkpoint_every][6][ld] predicted states of a segment
  double* adj = nullptr;    // [13][ld] xb vb ab jb, mb
  double* ab1 = nullptr;    // [6][ld] caller's acc/jerk adjoints (vjp_acc_jerk)
  double* mb = nullptr;     // adj's last array
  // Slots of the forward pass, [..][6][ld], or of the VJP, [..][7][ld]: each
  // pass's are summed by the kernel after it
  double* P = nullptr;
  JBody64* jb64 = nullptr;
  SymSub* jsub = nullptr;
  JAdj* jadj = nullptr;
  StepCtl* ctl = nullptr;
  int* status = nullptr;
  SymLaunch fwd, rev;
  bool have_forward = false;
};

namespace {

SymArgs sym_args(const nbody_adjoint* a, double* out) {
  SymArgs s{};
  s.n = a->n;
  s.ld = a->ld;
  s.eps2 = a->cfg.eps2;
  s.out = out;
  s.stride = static_cast<size_t>(a->ld);
  s.status = a->status;
  return s;
}

SoA7 own_state(const nbody_adjoint* a) {
  const size_t ld = a->ld;
  return SoA7{a->X, a->X + ld, a->X + 2 * ld, a->M, a->V, a->V + ld, a->V + 2 * ld};
}

// The forward's kernel and splits (the engine's choice) and the VJP's, of at most
// most_slots partial-sum slots each.
cudaError_t plan_passes(nbody_adjoint* a, int most_slots) {
  const bool fp64 = a->cfg.precision == NBODY_FP64;
  for (const bool wide : {false, true}) {
    if (a->n < sym_min_bodies(wide)) continue;
    const size_t smem = fp64 ? (wide ? sym_fp64_smem<4, kW, 2>() : sym_fp64_smem<2, kW, 4>())
                             : (wide ? sym_nf_smem<4, kW, 2>() : sym_nf_smem<2, kW, 1>());
    SymLaunch l;
    const cudaError_t e =
        l.plan(fp64 ? fwd_fp64(wide) : fwd_mixed(wide), smem, 32 * kW * (wide ? 4 : 2),
               fp64 ? kSymTile64 : wide ? 128 : 64, a->n, a->sms, sym_rate(fp64, wide),
               fp64 ? kSymTail64 : kSymTailNF, most_slots);
    if (e != cudaSuccess) return e;
    if (!wide || l.ms < a->fwd.ms) a->fwd = l;
  }
  return a->rev.plan(vjp_fn(), vjp_smem<2, kW>(), 32 * kW * 2, kVjpTile, a->n, a->sms, 3.3e8, kSymTail64,
                     most_slots);
}

nbody_status fwd_eval(nbody_adjoint* a, cudaStream_t st) {
  SymArgs s = sym_args(a, a->P);
  s.rows = own_state(a);
  AD_CUDA(a->fwd.launch(a->cfg.precision == NBODY_FP64 ? static_cast<const void*>(a->jb64) : a->jsub, s, st));
  return NBODY_OK;
}

nbody_status fwd_initial(nbody_adjoint* a, cudaStream_t st) {
  const size_t ld = a->ld;
  if (a->cfg.precision == NBODY_FP64)
    pack_kernel<<<(a->ld + kBlock - 1) / kBlock, kBlock, 0, st>>>(a->n, a->ld, own_state(a), a->jb64, nullptr);
  else
    sym_tile_kernel<false, false><<<a->ld / 64, 64, 0, st>>>(a->n, own_state(a), a->jsub);  // the caller's order
  AD_CUDA(cudaGetLastError());
  AD_TRY(fwd_eval(a, st));
  double* D = a->D;
  launch_reduce(st, 0, a->n, a->ld, a->fwd.slots(), a->P,
                SoA6{D, D + ld, D + 2 * ld, D + 3 * ld, D + 4 * ld, D + 5 * ld});
  AD_CUDA(cudaGetLastError());
  return NBODY_OK;
}

// One Hermite step; if xp_out, the predicted X/V ([6][ld]) go there too.
nbody_status fwd_step(nbody_adjoint* a, cudaStream_t st, double* xp_out) {
  if (a->cfg.precision == NBODY_FP64)
    AD_CUDA(launch_chained(predict_kernel, (a->n + kPredictBlock - 1) / kPredictBlock, kPredictBlock, 0, st,
                           a->n, a->ld, a->ctl, a->X, a->V, a->M, a->D, a->jb64, nullptr, nullptr, xp_out));
  else
    AD_CUDA(launch_chained(sym_tile_kernel<true, false>, a->ld / 64, 64, 0, st, a->n, own_state(a), a->jsub, a->ld,
                           a->X, a->V, a->D, a->ctl, nullptr, xp_out));
  AD_TRY(fwd_eval(a, st));
  launch_correct(st, a->n, a->ld, a->fwd.slots(), a->P, a->X, a->V, a->D, a->ctl, 1.0, true);
  AD_CUDA(cudaGetLastError());
  return NBODY_OK;
}

// The pass between two VJPs (adj_link_kernel).
nbody_status link(nbody_adjoint* a, cudaStream_t st, bool sum, bool post, AdjPack pack,
                  const double* XV = nullptr, const double* AB = nullptr) {
  constexpr int rows = kSumRows<8>;
  AD_CUDA(launch_chained(adj_link_kernel, (a->ld + rows - 1) / rows, kSumThreads, 0, st, a->n, a->ld,
                         a->cfg.dt, a->rev.slots(), sum, a->P, post, a->adj, a->mb,
                         static_cast<int>(pack), XV, a->M, AB, a->jadj));
  return NBODY_OK;
}

// Slots of the pair VJP at the packed records.
nbody_status vjp(nbody_adjoint* a, cudaStream_t st) {
  AD_CUDA(a->rev.launch(a->jadj, sym_args(a, a->P), st));
  return NBODY_OK;
}

bool all_local(const nbody_adjoint* a, const double* const* p, int count) {
  return std::all_of(p, p + count, [&](const double* q) {
    return !q || local_to(q, a->cfg.device, [](cudaPointerAttributes* at, const void* r) {
      return cudaPointerGetAttributes(at, r);
    });
  });
}

// The caller's `count` arrays (n each; null: zeros) into consecutive [ld]
// arrays, padding rows zero.  Arrays that are not this device's own memory go
// through the runtime's copies, which reach a peer's memory and refuse what
// they cannot read.
nbody_status copy_rows(nbody_adjoint* a, cudaStream_t st, const double* const* src, double* dst, int count) {
  if (!all_local(a, src, count)) {
    AD_CUDA(cudaMemsetAsync(dst, 0, sizeof(double) * a->ld * count, st));
    for (int k = 0; k < count; ++k)
      if (src[k])
        AD_CUDA(cudaMemcpyAsync(dst + static_cast<size_t>(k) * a->ld, src[k], sizeof(double) * a->n,
                                cudaMemcpyDeviceToDevice, st));
    return NBODY_OK;
  }
  GatherArgs g{};
  g.arrays = count;
  for (int k = 0; k < count; ++k) {
    g.src[k] = src[k];
    g.dst[k] = dst + static_cast<size_t>(k) * a->ld;
  }
  copy_rows_kernel<<<(a->ld + kBlock - 1) / kBlock, kBlock, 0, st>>>(a->n, a->ld, g, true);
  AD_CUDA(cudaGetLastError());
  return NBODY_OK;
}
// And back: consecutive [ld] arrays to the caller's.
nbody_status copy_out(nbody_adjoint* a, cudaStream_t st, const double* src, double* const* dst, int count) {
  if (!all_local(a, dst, count)) {
    for (int k = 0; k < count; ++k)
      AD_CUDA(cudaMemcpyAsync(dst[k], src + static_cast<size_t>(k) * a->ld, sizeof(double) * a->n,
                              cudaMemcpyDeviceToDevice, st));
    return NBODY_OK;
  }
  GatherArgs g{};
  g.arrays = count;
  for (int k = 0; k < count; ++k) {
    g.src[k] = src + static_cast<size_t>(k) * a->ld;
    g.dst[k] = dst[k];
  }
  copy_rows_kernel<<<(a->ld + kBlock - 1) / kBlock, kBlock, 0, st>>>(a->n, a->ld, g, false);
  AD_CUDA(cudaGetLastError());
  return NBODY_OK;
}

nbody_status set_ctl(nbody_adjoint* a, cudaStream_t st) {
  StepCtl c{};
  c.dt = a->cfg.dt;
  c.crit_bits = kPosInfBits;
  c.adaptive = 0;
  AD_CUDA(cudaMemcpyAsync(a->ctl, &c, sizeof c, cudaMemcpyHostToDevice, st));
  return NBODY_OK;
}

nbody_status check_status(nbody_adjoint* a, cudaStream_t st) {
  int h = 0;
  AD_CUDA(cudaMemcpyAsync(&h, a->status, sizeof h, cudaMemcpyDeviceToHost, st));
  AD_CUDA(cudaStreamSynchronize(st));
  if (h) {
    cudaMemsetAsync(a->status, 0, sizeof(int), st);
    return nbody_set_error(NBODY_ERR_TIMEOUT, "an adjoint pair-kernel wait exceeded its limit");
  }
  return NBODY_OK;
}

}  // namespace

extern "C" {

nbody_status nbody_adjoint_destroy(nbody_adjoint* a) {
  if (!a) return NBODY_OK;
  cudaSetDevice(a->cfg.device);
  cudaDeviceSynchronize();
  void* bufs[] = {a->state, a->ckpt, a->segxv, a->adj, a->ab1, a->P,
                  a->jb64, a->jsub, a->jadj, a->ctl, a->status};
  for (void* p : bufs) cudaFree(p);
  delete a;
  return NBODY_OK;
}

nbody_status nbody_adjoint_create(nbody_adjoint** out, const nbody_adjoint_config* cfg) {
  if (!out || !cfg) return nbody_set_error(NBODY_ERR_INVALID_ARG, "null argument");
  *out = nullptr;
  if (cfg->n < 1 || cfg->n > (1 << 22)) return nbody_set_error(NBODY_ERR_INVALID_ARG, "n = %d", cfg->n);
  if (!(cfg->eps2 >= 1e-30 && cfg->eps2 <= 1e30)) return nbody_set_error(NBODY_ERR_INVALID_ARG, "eps2 = %g", cfg->eps2);
  if (!(cfg->dt > 0)) return nbody_set_error(NBODY_ERR_INVALID_ARG, "dt must be > 0 (fixed step)");
  if (cfg->nsteps < 0 || cfg->checkpoint_every < 1)
    return nbody_set_error(NBODY_ERR_INVALID_ARG, "nsteps = %d, checkpoint_every = %d", cfg->nsteps, cfg->checkpoint_every);
  if (cfg->precision != NBODY_FP64 && cfg->precision != NBODY_MIXED)
    return nbody_set_error(NBODY_ERR_INVALID_ARG, "precision = %d", cfg->precision);
  if (cfg->precision == NBODY_MIXED && cfg->eps2 < kMinEps2Mixed)
    return nbody_set_error(NBODY_ERR_INVALID_ARG, "eps2 = %g below %g (mixed precision)", cfg->eps2,
                           kMinEps2Mixed);
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return nbody_set_error(NBODY_ERR_NO_DEVICE, "no CUDA device");
  if (cfg->device < 0 || cfg->device >= ndev) return nbody_set_error(NBODY_ERR_INVALID_ARG, "device %d", cfg->device);
  int major = 0;
  cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, cfg->device);
  if (major != 10) return nbody_set_error(NBODY_ERR_NO_DEVICE, "device %d is not sm_100", cfg->device);
  AD_CUDA(cudaSetDevice(cfg->device));
  std::unique_ptr<nbody_adjoint> a(new nbody_adjoint);
  a->cfg = *cfg;
  a->n = cfg->n;
  a->ld = (cfg->n + kPad - 1) / kPad * kPad;
  a->nseg = std::max(1, (cfg->nsteps + cfg->checkpoint_every - 1) / cfg->checkpoint_every);
  cudaDeviceGetAttribute(&a->sms, cudaDevAttrMultiProcessorCount, cfg->device);
  nbody_adjoint* r = a.get();
  auto body = [&]() -> nbody_status {
    const size_t ld = r->ld;
    const bool fp64 = cfg->precision == NBODY_FP64;
    AD_CUDA(cudaMalloc(&r->state, sizeof(double) * 13 * ld));
    AD_CUDA(cudaMemset(r->state, 0, sizeof(double) * 13 * ld));
    r->X = r->state;
    r->V = r->state + 3 * ld;
    r->M = r->state + 6 * ld;
    r->D = r->state + 7 * ld;
    AD_CUDA(cudaMalloc(&r->ckpt, sizeof(double) * 13 * ld * r->nseg));
    AD_CUDA(cudaMalloc(&r->segxv, sizeof(double) * 6 * ld * cfg->checkpoint_every));
    AD_CUDA(cudaMalloc(&r->adj, sizeof(double) * 13 * ld));
    r->mb = r->adj + 12 * ld;
    AD_CUDA(cudaMalloc(&r->ab1, sizeof(double) * 6 * ld));
    if (fp64) AD_CUDA(cudaMalloc(&r->jb64, sizeof(JBody64) * ld));
    else AD_CUDA(cudaMalloc(&r->jsub, sizeof(SymSub) * (ld / 64)));
    AD_CUDA(cudaMalloc(&r->jadj, sizeof(JAdj) * ld));
    AD_CUDA(cudaMalloc(&r->ctl, sizeof(StepCtl)));
    AD_CUDA(cudaMalloc(&r->status, sizeof(int)));
    AD_CUDA(cudaMemset(r->status, 0, sizeof(int)));
    // where memory is short, schedules of fewer blocks and splits
    for (int most = max_sym_slots(r->n);; most /= 2) {
      AD_CUDA(plan_passes(r, most));
      const size_t fields = std::max(6 * r->fwd.count(), 7 * r->rev.count());
      const cudaError_t e = cudaMalloc(&r->P, sizeof(double) * ld * fields);
      if (e == cudaSuccess) return NBODY_OK;
      r->P = nullptr;
      cudaGetLastError();
      if (e != cudaErrorMemoryAllocation || most <= 4) AD_CUDA(e);
    }
  };
  nbody_status s = body();
  if (s != NBODY_OK) {
    nbody_adjoint_destroy(a.release());
    return s;
  }
  *out = a.release();
  return NBODY_OK;
}

nbody_status nbody_adjoint_forward(nbody_adjoint* a, const double* x, const double* y, const double* z,
                                   const double* m, const double* vx, const double* vy,
                                   const double* vz, double* x1, double* y1, double* z1, double* vx1,
                                   double* vy1, double* vz1, void* stream) {
  TraceRange trace_("nbody_adjoint_forward");
  if (!a) return nbody_set_error(NBODY_ERR_INVALID_ARG, "null adjoint");
  const void* ptrs[13] = {x, y, z, m, vx, vy, vz, x1, y1, z1, vx1, vy1, vz1};
  for (auto p : ptrs)
    if (!p) return nbody_set_error(NBODY_ERR_INVALID_ARG, "null device array");
  AD_CUDA(cudaSetDevice(a->cfg.device));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const size_t ld = a->ld;
  const double* src[13] = {x, y, z, vx, vy, vz, m};  // the derivatives start at zero
  AD_TRY(copy_rows(a, st, src, a->state, 13));
  AD_TRY(set_ctl(a, st));
  AD_TRY(fwd_initial(a, st));
  const int K = a->cfg.checkpoint_every;
  for (int s = 0; s < a->cfg.nsteps; ++s) {
    if (s % K == 0)
      AD_CUDA(cudaMemcpyAsync(a->ckpt + static_cast<size_t>(s / K) * 13 * ld, a->state,
                              sizeof(double) * 13 * ld, cudaMemcpyDeviceToDevice, st));
    AD_TRY(fwd_step(a, st, nullptr));
  }
  if (a->cfg.nsteps == 0)
    AD_CUDA(cudaMemcpyAsync(a->ckpt, a->state, sizeof(double) * 13 * ld, cudaMemcpyDeviceToDevice, st));
  double* outs[6] = {x1, y1, z1, vx1, vy1, vz1};
  AD_TRY(copy_out(a, st, a->X, outs, 6));
  a->have_forward = true;
  return check_status(a, st);
}

nbody_status nbody_adjoint_backward(nbody_adjoint* a, const double* gx, const double* gy,
                                    const double* gz, const double* gvx, const double* gvy,
                                    const double* gvz, double* gx0, double* gy0, double* gz0,
                                    double* gvx0, double* gvy0, double* gvz0, double* gm,
                                    void* stream) {
  TraceRange trace_("nbody_adjoint_backward");
  if (!a) return nbody_set_error(NBODY_ERR_INVALID_ARG, "null adjoint");
  if (!a->have_forward) return nbody_set_error(NBODY_ERR_STATE, "backward before forward");
  const void* ptrs[13] = {gx, gy, gz, gvx, gvy, gvz, gx0, gy0, gz0, gvx0, gvy0, gvz0, gm};
  for (auto p : ptrs)
    if (!p) return nbody_set_error(NBODY_ERR_INVALID_ARG, "null device array");
  AD_CUDA(cudaSetDevice(a->cfg.device));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const size_t ld = a->ld;
  const int K = a->cfg.checkpoint_every, NS = a->cfg.nsteps;
  const double* g[13] = {gx, gy, gz, gvx, gvy, gvz};  // the rest of adj and mb start at zero
  AD_TRY(copy_rows(a, st, g, a->adj, 13));
  AD_TRY(set_ctl(a, st));
  for (int seg = a->nseg - 1; seg >= 0; --seg) {
    const int s0 = seg * K, s1 = std::min(NS, s0 + K);
    if (s1 <= s0) continue;
    AD_CUDA(cudaMemcpyAsync(a->state, a->ckpt + static_cast<size_t>(seg) * 13 * ld,
                            sizeof(double) * 13 * ld, cudaMemcpyDeviceToDevice, st));
    for (int s = s0; s < s1; ++s) AD_TRY(fwd_step(a, st, a->segxv + static_cast<size_t>(s - s0) * 6 * ld));
    for (int s = s1 - 1; s >= s0; --s) {
      const bool inside = s < s1 - 1;  // a VJP of this segment's next step to finish first
      AD_TRY(link(a, st, inside, inside, kPackStep, a->segxv + static_cast<size_t>(s - s0) * 6 * ld));
      AD_TRY(vjp(a, st));
    }
    AD_TRY(link(a, st, true, true, kPackNone));
  }
  // the initial acc/jerk: (a0, j0) = F(x_init, v_init, m), x_init in checkpoint 0
  AD_TRY(link(a, st, false, false, kPackFrom, a->ckpt, a->adj + 6 * ld));
  AD_TRY(vjp(a, st));
  AD_TRY(link(a, st, true, false, kPackNone));
  double* outs[6] = {gx0, gy0, gz0, gvx0, gvy0, gvz0};
  AD_TRY(copy_out(a, st, a->adj, outs, 6));
  AD_TRY(copy_out(a, st, a->mb, &gm, 1));
  return check_status(a, st);
}

nbody_status nbody_adjoint_vjp_acc_jerk(nbody_adjoint* a, const double* x, const double* y,
                                        const double* z, const double* m, const double* vx,
                                        const double* vy, const double* vz, const double* abx,
                                        const double* aby, const double* abz, const double* jbx,
                                        const double* jby, const double* jbz, double* gx,
                                        double* gy, double* gz, double* gvx, double* gvy,
                                        double* gvz, double* gm, void* stream) {
  if (!a) return nbody_set_error(NBODY_ERR_INVALID_ARG, "null adjoint");
  const void* ptrs[20] = {x, y, z, m, vx, vy, vz, abx, aby, abz, jbx, jby, jbz, gx, gy, gz, gvx, gvy, gvz, gm};
  for (auto p : ptrs)
    if (!p) return nbody_set_error(NBODY_ERR_INVALID_ARG, "null device array");
  AD_CUDA(cudaSetDevice(a->cfg.device));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  // inputs go to the segment buffer (state) and ab1 (adjoints); outputs via adj/mb
  const double* xv[6] = {x, y, z, vx, vy, vz};
  const double* ab[6] = {abx, aby, abz, jbx, jby, jbz};
  const double* zero[13] = {};
  AD_TRY(copy_rows(a, st, xv, a->segxv, 6));
  AD_TRY(copy_rows(a, st, ab, a->ab1, 6));
  AD_TRY(copy_rows(a, st, zero, a->adj, 13));
  AD_TRY(copy_rows(a, st, &m, a->M, 1));
  AD_TRY(link(a, st, false, false, kPackFrom, a->segxv, a->ab1));
  AD_TRY(vjp(a, st));
  AD_TRY(link(a, st, true, false, kPackNone));
  double* outs[6] = {gx, gy, gz, gvx, gvy, gvz};
  AD_TRY(copy_out(a, st, a->adj, outs, 6));
  AD_TRY(copy_out(a, st, a->mb, &gm, 1));
  a->have_forward = false;  // the state buffers now hold this call's inputs
  return check_status(a, st);
}

}  // extern "C"

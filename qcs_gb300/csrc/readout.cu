// readout.cu -- FP64-accumulated reductions, measurement, diffusion and shot
// sampling.
//
// Replaces the host loops of q_state_normalize (src/q_utils.c:44-119),
// qc_measure (src/qcs.c:237-284), qc_get_probability (:391-395),
// qc_find_most_likely_state (:464-478), qc_run_shots (:575-607) and
// q_apply_diffusion (src/q_gates.c:323-356).
//
// Precision plan (GB300 has little FP64 throughput): for complex64 states a
// thread forms |a|^2 (or re, im) in FP32 over 8 amplitudes, then adds that
// partial into FP64 accumulators; block and grid combination are FP64.  The
// grid is fixed per state size, so every reduction is deterministic.
// complex128 states use FP64 throughout.
//
// The last block of a reduction to finish combines the blocks' partials (in a
// fixed order) and leaves the result where it is wanted: in device memory, or
// straight in the state's pinned host buffer.  A call is then one kernel and
// one wait; a second kernel of one warp (10 us for 608 slots; 169 us where
// one thread walked them, for the argmax) and a copy back took longer than
// the reduction of a small state.
#include <type_traits>

#include "common.cuh"
#include "sampler.cuh"

namespace qcs {

enum { OP_NORM = 0, OP_MASK = 1, OP_SUM = 2 };

// Called by every thread of every block, after thread 0 has written the
// block's partial: true in the block that gets here last, which then sees
// every block's.  Leaves the counter at zero for the next launch.
__device__ __forceinline__ bool last_block(unsigned *count) {
  __shared__ bool last;
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(count, 1u) == gridDim.x - 1;
    if (last) {
      *count = 0;
      __threadfence();
    }
  }
  __syncthreads();
  return last;
}

// Lanes 0-15 get the warp's sum of a, the others that of b.
__device__ __forceinline__ double warp_sum2(double a, double b) {
  const bool up = (threadIdx.x & 16) != 0;
  double x = (up ? b : a) + __shfl_xor_sync(0xffffffffu, up ? a : b, 16);
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

// Two FP64 sums over the block; in warp 0, lane 0 gets that of a and lane 16
// that of b.  (Half the lanes for each: 8 additions in a row, where summing
// both, and two unused values, in every lane took 40 in the FP64 pipe: <Z> on
// 16 qubits 17.9 -> 14.0 us a call.)
__device__ __forceinline__ double block_sum2(double a, double b) {
  constexpr int kWarps = kReduceThreads / 32;
  static_assert(kWarps <= 16, "a lane of each half per warp");
  __shared__ double sh[2][kWarps];
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  double x = warp_sum2(a, b);
  if ((l & 15) == 0) sh[l >> 4][w] = x;
  __syncthreads();
  x = 0.0;
  if (w == 0) {
    x = (l & 15) < kWarps ? sh[l >> 4][l & 15] : 0.0;
#pragma unroll
    for (int o = kWarps / 2; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  }
  return x;
}

// The host waits for its call's number in result[kReady], written after
// everything else (by one thread, in step with those that wrote it): the
// kernel's end and the stream's take microseconds more to reach it.  The number
// tells this kernel's result from that of one before it whose call returned
// early, with an error.
constexpr int kReady = 7;
__device__ __forceinline__ void report(double *result, i64 call) {
  __threadfence_system();
  *(volatile i64 *)(result + kReady) = call;
}

// The block adds nblocks partials in a fixed order and writes the two sums.
// HOST: to the pinned buffer that the host reads.
template <bool HOST>
__device__ void sum_slots(const ReduceSlot *p, int nblocks, double *result, i64 call) {
  double a = 0.0, b = 0.0;
  for (int i = threadIdx.x; i < nblocks; i += blockDim.x) {
    const double2 x = __ldcg(reinterpret_cast<const double2 *>(p + i));
    a += x.x;
    b += x.y;
  }
  __syncthreads();
  const double x = block_sum2(a, b);
  if (threadIdx.x == 0) result[0] = x;
  if (threadIdx.x == 16) result[1] = x;
  __syncwarp();
  if (HOST && threadIdx.x == 0) report(result, call);
}

// Ends a reduction: the block's partial, then (last block) the total.
template <bool HOST>
__device__ __forceinline__ void reduce_end(double a, double b, ReduceSlot *slots, unsigned *count,
                                           double *result, i64 call) {
  const double x = block_sum2(a, b);
  if (threadIdx.x == 0) slots[blockIdx.x].a = x;
  if (threadIdx.x == 16) slots[blockIdx.x].b = x;
  __syncwarp();  // lane 16's partial, before thread 0 counts the block
  if (last_block(count)) sum_slots<HOST>(slots, gridDim.x, result, call);
}

template <int OP, typename R>
__device__ __forceinline__ void accum(i64 idx, R re, R im, int q, R &pa, R &pb) {
  if (OP == OP_NORM) {
    pa += re * re + im * im;
  } else if (OP == OP_MASK) {
    R p = re * re + im * im;
    if ((idx >> q) & 1) pb += p;
    else pa += p;
  } else {
    pa += re;
    pb += im;
  }
}

// complex64: units of two amplitudes (one 16-byte load), four units per
// step, FP32 within a step, FP64 across steps.  (Four blocks an SM is the grid;
// said so, the compiler keeps a step's four loads in flight: with 32 registers a
// pass over 28 qubits took 5 % longer.)
template <int OP>
__global__ void __launch_bounds__(kReduceThreads, 4)
    k_reduce_c64(const float4 *v, i64 units, int q, ReduceSlot *slots, unsigned *count,
                 double *result, i64 call) {
  grid_wait();
  const i64 nthr = (i64)gridDim.x * blockDim.x;
  double A = 0.0, B = 0.0;
  for (i64 u = (i64)blockIdx.x * blockDim.x + threadIdx.x; u < units; u += 4 * nthr) {
    float pa = 0.f, pb = 0.f;
    float4 x[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
      i64 uu = u + k * nthr;
      x[k] = uu < units ? v[uu] : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int k = 0; k < 4; k++) {
      i64 i0 = 2 * (u + k * nthr);
      if (OP == OP_MASK && q > 0) {
        // both amplitudes of the unit share bit q: one selection per unit
        const float p = (x[k].x * x[k].x + x[k].y * x[k].y) + (x[k].z * x[k].z + x[k].w * x[k].w);
        if ((i0 >> q) & 1) pb += p;
        else pa += p;
      } else {
        accum<OP>(i0, x[k].x, x[k].y, q, pa, pb);
        accum<OP>(i0 + 1, x[k].z, x[k].w, q, pa, pb);
      }
    }
    A += (double)pa;
    B += (double)pb;
  }
  reduce_end<OP != OP_SUM>(A, B, slots, count, result, call);
}

template <int OP>
__global__ void __launch_bounds__(kReduceThreads)
    k_reduce_c128(const double2 *v, i64 size, int q, ReduceSlot *slots, unsigned *count,
                  double *result, i64 call) {
  grid_wait();
  const i64 nthr = (i64)gridDim.x * blockDim.x;
  double A = 0.0, B = 0.0;
  for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < size; i += nthr) {
    double2 x = v[i];
    accum<OP, double>(i, x.x, x.y, q, A, B);
  }
  reduce_end<OP != OP_SUM>(A, B, slots, count, result, call);
}

// One block combines partials that another kernel left.
__global__ void __launch_bounds__(kReduceThreads)
    k_finalize(const ReduceSlot *p, int nblocks, double *result) {
  sum_slots<false>(p, nblocks, result, 0);
}

// Physical diffusion psi := 2*(S/N) - psi, fused with the sum of the new
// amplitudes (the sum is invariant in exact arithmetic; carrying the real
// sum of what was stored keeps a following phase flip's cached sum exact).
__global__ void __launch_bounds__(kReduceThreads)
    k_diffuse_c64(float4 *v, i64 units, double *S, double inv_n, ReduceSlot *slots,
                  unsigned *count) {
  const i64 nthr = (i64)gridDim.x * blockDim.x;
  const float tr = (float)(2.0 * (S[0] * inv_n));
  const float ti = (float)(2.0 * (S[1] * inv_n));
  double A = 0.0, B = 0.0;
  for (i64 u = (i64)blockIdx.x * blockDim.x + threadIdx.x; u < units; u += 4 * nthr) {
    float pa = 0.f, pb = 0.f;
    float4 x[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
      i64 uu = u + k * nthr;
      if (uu < units) x[k] = v[uu];
    }
#pragma unroll
    for (int k = 0; k < 4; k++) {
      i64 uu = u + k * nthr;
      if (uu < units) {
        float4 y = make_float4(tr - x[k].x, ti - x[k].y, tr - x[k].z, ti - x[k].w);
        v[uu] = y;
        pa += y.x + y.z;
        pb += y.y + y.w;
      }
    }
    A += (double)pa;
    B += (double)pb;
  }
  reduce_end<false>(A, B, slots, count, S, 0);  // every block has read S by now
}

__global__ void __launch_bounds__(kReduceThreads)
    k_diffuse_c128(double2 *v, i64 size, double *S, double inv_n, ReduceSlot *slots,
                   unsigned *count) {
  const i64 nthr = (i64)gridDim.x * blockDim.x;
  const double tr = 2.0 * (S[0] * inv_n);
  const double ti = 2.0 * (S[1] * inv_n);
  double A = 0.0, B = 0.0;
  for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < size; i += nthr) {
    double2 x = v[i];
    double2 y = make_double2(__dsub_rn(tr, x.x), __dsub_rn(ti, x.y));
    v[i] = y;
    A += y.x;
    B += y.y;
  }
  reduce_end<false>(A, B, slots, count, S, 0);
}

// The reference's diffusion (src/q_gates.c:334-355): mean := S/|S| when
// |S| > 1e-10, dst := 2*mean - src (dst is the swapped-in buffer).
template <typename C>
__global__ void __launch_bounds__(kSweepThreads)
    k_diffuse_reference(C *dst, const C *src, i64 size, const double *S) {
  double mr = S[0], mi = S[1];
  double mag = sqrt(__dadd_rn(__dmul_rn(mr, mr), __dmul_rn(mi, mi)));
  if (mag > 1e-10) {
    mr /= mag;
    mi /= mag;
  }
  const C two = make_c<C>(2.0 * mr, 2.0 * mi);
  const i64 nthr = (i64)gridDim.x * blockDim.x;
  for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < size; i += nthr) {
    C x = src[i];
    dst[i] = make_c<C>((double)(two.x - x.x), (double)(two.y - x.y));
  }
}

// Collapse after a measurement: amplitudes whose bit q differs from the
// outcome become 0, the others are multiplied by `scale` when do_scale.
// complex64 in units of two amplitudes (one 16-byte access), four units in
// flight per thread: for q >= 1 both amplitudes of a unit share bit q, so
// the discarded half is written without being read, and the kept half is
// read only when it is rescaled; for q = 0 each unit holds one of each.
__global__ void __launch_bounds__(kReduceThreads)
    k_collapse_c64(float4 *v, i64 units, int q, int outcome, float scale, int do_scale) {
  const i64 nthr = (i64)gridDim.x * blockDim.x;
  for (i64 u = (i64)blockIdx.x * blockDim.x + threadIdx.x; u < units; u += 4 * nthr) {
    float4 x[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const i64 uu = u + k * nthr;
      const bool keep = q == 0 || (int)(((2 * uu) >> q) & 1) == outcome;
      if (uu < units && keep && (q == 0 || do_scale)) x[k] = v[uu];
    }
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const i64 uu = u + k * nthr;
      if (uu >= units) continue;
      if (q == 0) {
        const float s = do_scale ? scale : 1.f;
        v[uu] = outcome == 0 ? make_float4(x[k].x * s, x[k].y * s, 0.f, 0.f)
                             : make_float4(0.f, 0.f, x[k].z * s, x[k].w * s);
      } else if ((int)(((2 * uu) >> q) & 1) == outcome) {
        if (do_scale)
          v[uu] = make_float4(x[k].x * scale, x[k].y * scale, x[k].z * scale, x[k].w * scale);
      } else {
        v[uu] = make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
  }
}

// complex128: one amplitude (16 bytes) per unit, four in flight per thread.
__global__ void __launch_bounds__(kReduceThreads)
    k_collapse_c128(double2 *v, i64 size, int q, int outcome, double scale, int do_scale) {
  const i64 nthr = (i64)gridDim.x * blockDim.x;
  for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < size; i += 4 * nthr) {
    double2 x[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const i64 j = i + k * nthr;
      if (j < size && do_scale && (int)((j >> q) & 1) == outcome) x[k] = v[j];
    }
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const i64 j = i + k * nthr;
      if (j >= size) continue;
      if ((int)((j >> q) & 1) == outcome) {
        if (do_scale) v[j] = make_double2(x[k].x * scale, x[k].y * scale);
      } else {
        v[j] = make_double2(0.0, 0.0);
      }
    }
  }
}

// One amplitude, to the host (8 us a call, and 3 less behind
// another kernel, than a copy and the stream's end: 9 and 13).
template <typename C>
__global__ void k_peek(const C *v, i64 index, double *result, i64 call) {
  grid_wait();
  const C x = v[index];
  result[0] = x.x;
  result[1] = x.y;
  report(result, call);
}

// Every qubit of a small state measured in one block, the state in shared
// memory: per qubit P(0) and P(1) (FP32 squares of two adjacent amplitudes,
// summed in FP64; complex128 in FP64), the outcome of its draw, the collapse.
// A thread keeps its pairs of amplitudes, so a qubit's collapse and the next
// one's sums are one pass.  Bound by the FP64 pipe's latency and width (two
// lanes per clock: hence few warps, and sums that split the lanes between P(0)
// and P(1)).  10 qubits: 25 us with the wait; a measurement that
// returns to the host for its outcome takes a reduction, a wait and a
// collapse, 18 us a qubit.  Above 128 KB one SM no longer holds the state.
constexpr int kMeasureMaxBytes = 128 << 10;
constexpr int kMeasureMaxQubits = 14;
constexpr int kMeasureThreads = 512;
struct MeasureDraws { double r[kMeasureMaxQubits]; };

template <typename C>
__global__ void __launch_bounds__(kMeasureThreads)
    k_measure_all(C *v, int n, const __grid_constant__ MeasureDraws draws, double *outcomes,
                  i64 call) {
  using R = decltype(C::x);
  constexpr int kWarps = kMeasureThreads / 32;  // 16: a lane each for P(0) and P(1)
  extern __shared__ __align__(16) unsigned char measure_smem[];
  C *S = reinterpret_cast<C *>(measure_smem);
  __shared__ double part[2][kWarps];
  __shared__ R s_scale;
  __shared__ int s_out;
  const int size = 1 << n, T = blockDim.x, warps = T / 32;
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  grid_wait();
  int bits = 0;  // thread 0: the outcomes so far
  int o = 0;     // the last qubit's outcome and scale
  R s = (R)1;
  for (int q = 0; q <= n; q++) {
    double A = 0.0, B = 0.0;
    for (int i = 2 * threadIdx.x; i < size; i += 2 * T) {  // n >= 1
      C x, y;
      if (q == 0) {
        x = v[i];
        y = v[i + 1];
      } else {  // collapsed
        x = S[i];
        y = S[i + 1];
        const bool kx = ((i >> (q - 1)) & 1) == o, ky = (((i + 1) >> (q - 1)) & 1) == o;
        x.x = kx ? x.x * s : (R)0;
        x.y = kx ? x.y * s : (R)0;
        y.x = ky ? y.x * s : (R)0;
        y.y = ky ? y.y * s : (R)0;
      }
      if (q == n) {
        v[i] = x;
        v[i + 1] = y;
        continue;
      }
      S[i] = x;
      S[i + 1] = y;
      const R px = x.x * x.x + x.y * x.y, py = y.x * y.x + y.y * y.y;
      if (q == 0) {
        A += (double)px;
        B += (double)py;
      } else if ((i >> q) & 1) {
        B += (double)(px + py);
      } else {
        A += (double)(px + py);
      }
    }
    if (q == n) break;
    const double sum = warp_sum2(A, B);
    if ((l & 15) == 0) part[l >> 4][w] = sum;
    __syncthreads();
    if (w == 0) {
      double x = (l & 15) < warps ? part[l >> 4][l & 15] : 0.0;
#pragma unroll
      for (int k = kWarps / 2; k > 0; k >>= 1) x += __shfl_xor_sync(0xffffffffu, x, k);
      const double other = __shfl_xor_sync(0xffffffffu, x, 16);
      if (l == 0) {
        const int out = draws.r[q] <= x ? 0 : 1;
        const double kept = out ? other : x;
        s_scale = kept > 1e-12 && kept != 1.0 ? (R)(1.0 / sqrt(kept)) : (R)1;
        s_out = out;
        bits |= out << q;
      }
    }
    __syncthreads();
    o = s_out;
    s = s_scale;
  }
  __syncthreads();  // the state is written
  if (threadIdx.x == 0) {
    outcomes[0] = (double)bits;
    report(outcomes, call);
  }
}

template <typename C, typename R>
__global__ void __launch_bounds__(kSweepThreads) k_scale(C *v, i64 size, R scale) {
  const i64 nthr = (i64)gridDim.x * blockDim.x;
  for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < size; i += nthr) {
    C x = v[i];
    x.x *= scale;
    x.y *= scale;
    v[i] = x;
  }
}

// ---- argmax ---------------------------------------------------------------
// Order: larger value first, then smaller index -- the first strict maximum
// of the reference's ascending scan.  NaN never wins.
template <typename R>
__device__ __forceinline__ bool better(R v, i64 i, R bv, i64 bi) {
  return v > bv || (v == bv && i < bi);
}

// The best (value, index) pair over the block, in thread 0.
template <typename R>
__device__ __forceinline__ void block_best(R &bv, i64 &bi) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const R ov = __shfl_xor_sync(0xffffffffu, bv, o);
    const i64 oi = __shfl_xor_sync(0xffffffffu, bi, o);
    if (better(ov, oi, bv, bi)) {
      bv = ov;
      bi = oi;
    }
  }
  __shared__ R sv[kReduceThreads / 32];
  __shared__ i64 si[kReduceThreads / 32];
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) {
    sv[w] = bv;
    si[w] = bi;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int k = 1; k < (int)(blockDim.x >> 5); k++)
      if (better(sv[k], si[k], bv, bi)) {
        bv = sv[k];
        bi = si[k];
      }
  }
}

// Ends an argmax: the block's best, then (last block) the best of all.
template <typename R>
__device__ __forceinline__ void argmax_end(R bv, i64 bi, ReduceSlot *slots, unsigned *count,
                                           double *result, i64 call) {
  block_best(bv, bi);
  if (threadIdx.x == 0) {
    slots[blockIdx.x].a = (double)bv;
    slots[blockIdx.x].b = (double)bi;
  }
  if (!last_block(count)) return;
  double v = -1.0;
  i64 at = 1LL << 62;
  for (int k = threadIdx.x; k < (int)gridDim.x; k += blockDim.x) {
    const double2 x = __ldcg(reinterpret_cast<const double2 *>(slots + k));
    if (better(x.x, (i64)x.y, v, at)) {
      v = x.x;
      at = (i64)x.y;
    }
  }
  block_best(v, at);
  if (threadIdx.x == 0) {
    result[0] = v;
    result[1] = (double)at;
    report(result, call);
  }
}

template <typename C, typename R>
__global__ void __launch_bounds__(kReduceThreads)
    k_argmax(const C *v, i64 size, ReduceSlot *slots, unsigned *count, double *result, i64 call) {
  const i64 nthr = (i64)gridDim.x * blockDim.x;
  R bv = (R)-1;
  i64 bi = size;
  for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < size; i += nthr) {
    C x = v[i];
    R p = (x.x * x.x) + (x.y * x.y);
    if (better(p, i, bv, bi)) {
      bv = p;
      bi = i;
    }
  }
  argmax_end(bv, bi, slots, count, result, call);
}

// complex64: units of two amplitudes (one 16-byte load), four in flight per
// thread; the same order (larger |a|^2, then smaller index) makes the result
// independent of which thread saw which amplitude.
__global__ void __launch_bounds__(kReduceThreads)
    k_argmax_c64(const float4 *v, i64 units, ReduceSlot *slots, unsigned *count,
                 double *result, i64 call) {
  const i64 nthr = (i64)gridDim.x * blockDim.x;
  float bv = -1.f;
  i64 bi = 2 * units;
  for (i64 u = (i64)blockIdx.x * blockDim.x + threadIdx.x; u < units; u += 4 * nthr) {
    float4 x[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const i64 uu = u + k * nthr;
      if (uu < units) x[k] = v[uu];
    }
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const i64 uu = u + k * nthr;
      if (uu >= units) continue;
      const float p0 = (x[k].x * x[k].x) + (x[k].y * x[k].y);
      const float p1 = (x[k].z * x[k].z) + (x[k].w * x[k].w);
      if (better(p0, 2 * uu, bv, bi)) {
        bv = p0;
        bi = 2 * uu;
      }
      if (better(p1, 2 * uu + 1, bv, bi)) {
        bv = p1;
        bi = 2 * uu + 1;
      }
    }
  }
  argmax_end(bv, bi, slots, count, result, call);
}

// ---- shot sampling: sampler.cuh -------------------------------------------------

// ---- host side -----------------------------------------------------------------

// Blocks of a reduction over `work` items, one per thread and step: the
// device's fixed reduction grid, or as many as have work.  (A grid that small
// gives each thread one item, so the partial sums are those of the full grid.)
static int reduce_grid(const qcs_cuda_state *s, i64 work) {
  const i64 need = (work + kReduceThreads - 1) / kReduceThreads;
  return (int)(need < 1 ? 1 : need < s->dev.reduce_blocks ? need : s->dev.reduce_blocks);
}

// Waits for a result that a kernel wrote to the pinned host buffer.
static int wait_result(qcs_cuda_state *s, size_t bytes, const char *what) {
  s->d2h_bytes += (long long)bytes;
  return check_cuda(cudaStreamSynchronize(s->stream), what);
}

// The same for a kernel that ends with report(): by watching for its call's
// number, a few microseconds sooner than the stream is known to be done (<Z> on 16
// qubits 14.0 -> 12.2 us a call).  (A profiled launch's closing event is waited
// for too.)
static i64 next_call(qcs_cuda_state *s) { return ++s->calls; }
static int wait_report(qcs_cuda_state *s, i64 call, size_t bytes, const char *what) {
  if (!s->prof) {
    const i64 *ready = (const i64 *)(s->h_result + kReady);
    // 0.34 ms on the Grace host of a GB300, 1 to 2 ms on x86 hosts; a longer wait is
    // left to the stream
    for (int i = 0; i < (1 << 20); i++)
      if (__atomic_load_n(ready, __ATOMIC_ACQUIRE) == call) {
        s->d2h_bytes += (long long)bytes;
        return QCS_CUDA_OK;
      }
  }
  return wait_result(s, bytes, what);
}

// Result in the pinned buffer (res != null), or, for the sum, on the device.
static int reduce(qcs_cuda_state *s, int op, int q, double *res, int nres) {
  const bool c128 = s->prec == QCS_CUDA_C128;
  const double Ns = (double)s->size * (c128 ? 16 : 8);
  double *dst = op == OP_SUM ? s->d_result + 4 : s->h_result_dev;
  const i64 work = c128 ? s->size : s->size / 2;
  const int grid = reduce_grid(s, work);
  const i64 call = next_call(s);
  prof_begin(s);
  auto go = [&](auto opc) {
    constexpr int OP = decltype(opc)::value;
    if (c128)
      launch_next(sweep_early(s, grid), k_reduce_c128<OP>, grid, kReduceThreads, 0, s->stream,
                  (const double2 *)s->vec, work, q, s->d_partials, s->d_count, dst,
                  call);
    else
      launch_next(sweep_early(s, grid), k_reduce_c64<OP>, grid, kReduceThreads, 0, s->stream,
                  (const float4 *)s->vec, work, q, s->d_partials, s->d_count, dst,
                  call);
  };
  if (op == OP_NORM) go(std::integral_constant<int, OP_NORM>());
  else if (op == OP_MASK) go(std::integral_constant<int, OP_MASK>());
  else go(std::integral_constant<int, OP_SUM>());
  int rc = launched(s, KC_REDUCE, Ns, "reduce");
  if (rc || !res) return rc;
  rc = wait_report(s, call, 4 * sizeof(double), "reduce sync");
  if (rc) return rc;
  for (int i = 0; i < nres; i++) res[i] = s->h_result[i];
  return QCS_CUDA_OK;
}

static int scale_state(qcs_cuda_state *s, double inv) {
  int g = grid_for(s->size, kSweepThreads, s->dev, 8);
  prof_begin(s);
  if (s->prec == QCS_CUDA_C128)
    k_scale<double2, double><<<g, kSweepThreads, 0, s->stream>>>((double2 *)s->vec, s->size, inv);
  else
    k_scale<float2, float><<<g, kSweepThreads, 0, s->stream>>>((float2 *)s->vec, s->size, (float)inv);
  return launched(s, KC_COLLAPSE, 2.0 * s->size * (s->prec == QCS_CUDA_C128 ? 16 : 8),
                  "normalize");
}

int diffusion(qcs_cuda_state *s) {
  const DeviceInfo &d = s->dev;
  const double Ns = (double)s->size * (s->prec == QCS_CUDA_C128 ? 16 : 8);
  int rc;
  if (s->sem == QCS_CUDA_REFERENCE) {
    rc = reduce(s, OP_SUM, 0, nullptr, 0);
    if (rc) return rc;
    void *src = s->vec;
    s->vec = s->scratch;
    s->scratch = src;
    int g = grid_for(s->size, kSweepThreads, d, 8);
    prof_begin(s);
    if (s->prec == QCS_CUDA_C128)
      k_diffuse_reference<double2><<<g, kSweepThreads, 0, s->stream>>>(
          (double2 *)s->vec, (const double2 *)src, s->size, s->d_result + 4);
    else
      k_diffuse_reference<float2><<<g, kSweepThreads, 0, s->stream>>>(
          (float2 *)s->vec, (const float2 *)src, s->size, s->d_result + 4);
    invalidate_sum(s);
    return launched(s, KC_DIFFUSE, 2 * Ns, "diffusion");
  }
  if (!s->sum_valid) {
    rc = reduce(s, OP_SUM, 0, nullptr, 0);
    if (rc) return rc;
  }
  double inv_n = ldexp(1.0, -s->n);
  prof_begin(s);
  if (s->prec == QCS_CUDA_C128)
    k_diffuse_c128<<<reduce_grid(s, s->size), kReduceThreads, 0, s->stream>>>(
        (double2 *)s->vec, s->size, s->d_result + 4, inv_n, s->d_partials, s->d_count);
  else
    k_diffuse_c64<<<reduce_grid(s, s->size / 2), kReduceThreads, 0, s->stream>>>(
        (float4 *)s->vec, s->size / 2, s->d_result + 4, inv_n, s->d_partials, s->d_count);
  rc = launched(s, KC_DIFFUSE, 2 * Ns, "diffusion");
  if (rc) return rc;
  s->sum_valid = 1;
  return QCS_CUDA_OK;
}

int norm_sq(qcs_cuda_state *s, double *out) { return reduce(s, OP_NORM, 0, out, 1); }

// The cached amplitude sum, computed now unless it is valid.
int ensure_sum(qcs_cuda_state *s) {
  if (s->sum_valid) return QCS_CUDA_OK;
  int rc = reduce(s, OP_SUM, 0, nullptr, 0);
  if (!rc) s->sum_valid = 1;
  return rc;
}

// A kernel left per-part sums of the new amplitudes in d_partials[0..nslots):
// combine them (fixed order) into the cached sum.
int finalize_sum(qcs_cuda_state *s, int nslots) {
  prof_begin(s);
  k_finalize<<<1, kReduceThreads, 0, s->stream>>>(s->d_partials, nslots, s->d_result + 4);
  int rc = launched(s, KC_OTHER, nslots * 32.0, "sum finalize");
  if (!rc) s->sum_valid = 1;
  return rc;
}

}  // namespace qcs

using namespace qcs;

extern "C" {

int qcs_cuda_diffusion(qcs_cuda_state *s) {
  QCS_CHECK_STATE(s);
  return diffusion(s);
}

int qcs_cuda_norm_sq(qcs_cuda_state *s, double *out) {
  QCS_CHECK_STATE(s);
  if (!out) return set_error(QCS_CUDA_EINVAL, "null out");
  return norm_sq(s, out);
}

int qcs_cuda_normalize(qcs_cuda_state *s) {
  QCS_CHECK_STATE(s);
  double total;
  int rc = norm_sq(s, &total);
  if (rc) return rc;
  if (total > 1e-12 && total != 1.0) {
    invalidate_sum(s);
    return scale_state(s, 1.0 / sqrt(total));
  }
  return QCS_CUDA_OK;
}

int qcs_cuda_prob_zero(qcs_cuda_state *s, int qubit, double *p0) {
  QCS_CHECK_STATE(s);
  if (!p0) return set_error(QCS_CUDA_EINVAL, "null out");
  if (qubit < 0 || qubit >= s->n) return set_error(QCS_CUDA_EINVAL, "qubit %d out of range", qubit);
  double r[2];
  int rc = reduce(s, OP_MASK, qubit, r, 2);
  if (!rc) *p0 = r[0];
  return rc;
}

int qcs_cuda_expect_z(qcs_cuda_state *s, int qubit, double *out) {
  QCS_CHECK_STATE(s);
  if (!out) return set_error(QCS_CUDA_EINVAL, "null out");
  if (qubit < 0 || qubit >= s->n) return set_error(QCS_CUDA_EINVAL, "qubit %d out of range", qubit);
  double r[2];
  int rc = reduce(s, OP_MASK, qubit, r, 2);
  if (!rc) *out = r[0] - r[1];
  return rc;
}

int qcs_cuda_measure(qcs_cuda_state *s, int qubit, double random_val, int *outcome) {
  QCS_CHECK_STATE(s);
  if (!outcome) return set_error(QCS_CUDA_EINVAL, "null out");
  if (qubit < 0 || qubit >= s->n) return set_error(QCS_CUDA_EINVAL, "qubit %d out of range", qubit);
  double r[2];
  int rc = reduce(s, OP_MASK, qubit, r, 2);
  if (rc) return rc;
  int o = (random_val <= r[0]) ? 0 : 1;
  double kept = o ? r[1] : r[0];
  int do_scale = (kept > 1e-12 && kept != 1.0);
  double inv = do_scale ? 1.0 / sqrt(kept) : 1.0;
  prof_begin(s);
  if (s->prec == QCS_CUDA_C128)
    k_collapse_c128<<<reduce_grid(s, s->size), kReduceThreads, 0, s->stream>>>(
        (double2 *)s->vec, s->size, qubit, o, inv, do_scale);
  else
    k_collapse_c64<<<reduce_grid(s, s->size / 2), kReduceThreads, 0, s->stream>>>(
        (float4 *)s->vec, s->size / 2, qubit, o, (float)inv, do_scale);
  invalidate_sum(s);
  rc = launched(s, KC_COLLAPSE, 1.5 * s->size * (s->prec == QCS_CUDA_C128 ? 16 : 8),
                "measure collapse");
  if (rc) return rc;
  *outcome = o;
  return QCS_CUDA_OK;
}

int qcs_measure_all(qcs_cuda_state *s, const double *random_vals, int *outcomes) {
  QCS_CHECK_STATE(s);
  const bool c128 = s->prec == QCS_CUDA_C128;
  const size_t bytes = (size_t)s->size * (c128 ? 16 : 8);
  if (s->n > kMeasureMaxQubits || bytes > (size_t)kMeasureMaxBytes) return QCS_CUDA_EUNSUP;
  MeasureDraws draws = {};
  for (int q = 0; q < s->n; q++) draws.r[q] = random_vals[q];
  const int pairs = (int)(s->size / 2);
  // four pairs a thread: fewer warps share the FP64 pipe
  const int threads = pairs < 128 ? 32 : pairs < 4 * kMeasureThreads ? pairs / 4 : kMeasureThreads;
  int rc = QCS_CUDA_OK;
  if (bytes > (48 << 10)) {  // the launch's default limit
    const void *k = c128 ? (const void *)k_measure_all<double2> : (const void *)k_measure_all<float2>;
    rc = check_cuda(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         kMeasureMaxBytes),
                    "cudaFuncSetAttribute(measure)");
  }
  // It collapses the state: not launched while an error is pending that
  // launched() would report as its own.
  if (!rc) rc = check_launch("measure all");
  if (rc) return rc;
  const i64 call = next_call(s);
  prof_begin(s);
  if (c128)
    launch_next(true, k_measure_all<double2>, 1, threads, bytes, s->stream, (double2 *)s->vec, s->n,
                draws, s->h_result_dev, call);
  else
    launch_next(true, k_measure_all<float2>, 1, threads, bytes, s->stream, (float2 *)s->vec, s->n,
                draws, s->h_result_dev, call);
  invalidate_sum(s);
  rc = launched(s, KC_COLLAPSE, 2.0 * bytes, "measure all");
  if (!rc) rc = wait_report(s, call, sizeof(double), "measure sync");
  if (rc) return rc;
  const int bits = (int)s->h_result[0];
  for (int q = 0; q < s->n; q++) outcomes[q] = (bits >> q) & 1;
  return QCS_CUDA_OK;
}

int qcs_cuda_probability(qcs_cuda_state *s, long long index, double *p) {
  QCS_CHECK_STATE(s);
  if (!p) return set_error(QCS_CUDA_EINVAL, "null out");
  if (index < 0 || index >= s->size) {
    *p = 0.0;  // qc_get_probability returns 0.0 out of range (src/qcs.c:392-393)
    return QCS_CUDA_OK;
  }
  const size_t bytes = s->prec == QCS_CUDA_C128 ? 16 : 8;
  const i64 call = next_call(s);
  prof_begin(s);
  if (s->prec == QCS_CUDA_C128)
    launch_next(true, k_peek<double2>, 1, 1, 0, s->stream, (const double2 *)s->vec, (i64)index,
                s->h_result_dev, call);
  else
    launch_next(true, k_peek<float2>, 1, 1, 0, s->stream, (const float2 *)s->vec, (i64)index,
                s->h_result_dev, call);
  int rc = launched(s, KC_OTHER, (double)bytes, "probability");
  if (!rc) rc = wait_report(s, call, bytes, "probability sync");
  if (rc) return rc;
  const double re = s->h_result[0], im = s->h_result[1];
  *p = (re * re) + (im * im);
  return QCS_CUDA_OK;
}

int qcs_cuda_argmax(qcs_cuda_state *s, long long *index, double *prob) {
  QCS_CHECK_STATE(s);
  if (!index) return set_error(QCS_CUDA_EINVAL, "null out");
  const bool pairs = s->prec == QCS_CUDA_C64;  // n >= 1: at least one pair
  const int grid = reduce_grid(s, pairs ? s->size / 2 : s->size);
  const i64 call = next_call(s);
  prof_begin(s);
  if (pairs)
    k_argmax_c64<<<grid, kReduceThreads, 0, s->stream>>>(
        (const float4 *)s->vec, s->size / 2, s->d_partials, s->d_count, s->h_result_dev, call);
  else
    k_argmax<double2, double><<<grid, kReduceThreads, 0, s->stream>>>(
        (const double2 *)s->vec, s->size, s->d_partials, s->d_count, s->h_result_dev, call);
  int rc = launched(s, KC_REDUCE, (double)s->size * (s->prec == QCS_CUDA_C128 ? 16 : 8),
                    "argmax");
  if (!rc) rc = wait_report(s, call, 2 * sizeof(double), "argmax sync");
  if (rc) return rc;
  *index = (long long)s->h_result[1];
  if (prob) return qcs_cuda_probability(s, *index, prob);
  return QCS_CUDA_OK;
}

int qcs_cuda_sample(qcs_cuda_state *s, const double *random_vals, int shots,
                    long long *out_index) {
  QCS_CHECK_STATE(s);
  if (shots < 0 || (shots > 0 && (!random_vals || !out_index)))
    return set_error(QCS_CUDA_EINVAL, "bad shot arguments");
  if (shots == 0) return QCS_CUDA_OK;
  int rc = ensure_sample_scratch(s, shots);
  if (rc) return rc;
  const i64 tile = s->size / s->n_tiles;
  const DeviceInfo &d = s->dev;
  int G = 1;
  i64 per = 1;
  smp_ranges(s->n_tiles, d.num_sms, d.num_sms * 8, &G, &per);
  double *in = s->d_tile_prefix, *boff = s->d_tile_prefix + s->n_tiles;
  const double sb = s->prec == QCS_CUDA_C128 ? 16 : 8;
  prof_begin(s);
  if (s->prec == QCS_CUDA_C128)
    k_smp_tile_sums<double2><<<G, kSampleThreads, 0, s->stream>>>(
        (const double2 *)s->vec, tile, s->n_tiles, per, in, boff, s->d_count);
  else
    k_smp_tile_sums<float2><<<G, kSampleThreads, 0, s->stream>>>(
        (const float2 *)s->vec, tile, s->n_tiles, per, in, boff, s->d_count);
  rc = launched(s, KC_SAMPLE, s->size * sb, "sample tile sums");
  if (rc) return rc;
  // the kernel reads the draws from, and writes the samples to, pinned host
  // memory: 8 bytes a shot beside the 64 KB it scans for it
  memcpy(s->h_draws, random_vals, (size_t)shots * sizeof(double));
  s->h2d_bytes += (long long)((size_t)shots * sizeof(double));
  int threads = 256;
  int blocks = (int)(((i64)shots * 32 + threads - 1) / threads);
  if (blocks > d.num_sms * 16) blocks = d.num_sms * 16;
  prof_begin(s);
  if (s->prec == QCS_CUDA_C128)
    k_smp_sample<double2><<<blocks, threads, 0, s->stream>>>(
        (const double2 *)s->vec, tile, s->n_tiles, per, in, boff, G, s->h_draws_dev, shots,
        s->h_samples_dev);
  else
    k_smp_sample<float2><<<blocks, threads, 0, s->stream>>>(
        (const float2 *)s->vec, tile, s->n_tiles, per, in, boff, G, s->h_draws_dev, shots,
        s->h_samples_dev);
  rc = launched(s, KC_SAMPLE, (double)shots * tile * sb, "sample");
  if (!rc) rc = wait_result(s, (size_t)shots * sizeof(i64), "sample sync");
  if (rc) return rc;
  memcpy(out_index, s->h_samples, (size_t)shots * sizeof(i64));
  return QCS_CUDA_OK;
}

}  // extern "C"

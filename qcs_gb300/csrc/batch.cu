// batch.cu -- many independent circuits in one persistent kernel launch.
//
// The reference simulates one circuit per t_q_circuit, every gate a full
// sweep (src/qcs.c:159-228), and reads results with qc_measure/qc_run_shots
// (:237-284, :575-607).  A batch of thousands of small-to-medium circuits
// (10..22 qubits) is launch-bound that way.  Here one persistent kernel takes
// the whole batch:
//
//  * CTAs pull instances from an atomic queue, largest first (the order is
//    part of the tuned schedule);
//  * an instance of at most `tile_q` qubits lives entirely in shared memory:
//    |0...0> is built there, its gates run there, and <Z_0> and the shots
//    are computed there -- it never touches HBM;
//  * gates run in register groups: the gates of a stage are cut into groups
//    on at most 4 or 5 tile bits, and one pass over shared memory applies a
//    whole group, each thread holding the 16 or 32 amplitudes of one setting
//    of the other bits in registers (one pass per group instead of one per
//    gate; tile_regs.cuh);
//  * a larger instance lives in a slot of global memory and runs in
//    stages: a stage is a set of tile_q qubits and the gates acting inside
//    it; for every tile (one setting of the other qubits) the CTA gathers the
//    2^tile_q amplitudes into shared memory with coalesced runs, applies the
//    stage's gates there and scatters them back, so a stage costs one read
//    and one write of the state however many gates it holds; the tiles are
//    handed out by tickets to every CTA that comes free;
//  * <Z_0> is accumulated in FP64 (of FP32 squares) and each shot is drawn
//    from a counter-based generator (splitmix64 of seed, instance, shot) and
//    mapped to an index by binary searches over running sums in FP64, then
//    the amplitudes of the block found.
//
// The run is captured once into a CUDA graph (queue reset, kernel, result
// copies) and replayed; new angles only rewrite the pinned gate table the
// graph's upload node reads.  The schedule (threads per CTA, tile size,
// CTAs per SM, instance order) comes from qcs_cuda_batch_autotune, which
// times the candidates on the batch itself.
//
// Measured (default schedule, 1024 shots): 384 instances of 10-22 qubits, 4-16
// layers 110 -> 48 ms against the kernel that kept a thread's amplitudes in
// C++ variables, read its gates from global memory, shared an instance among
// fixed CTAs and scanned 4096 amplitudes a shot; 608 of 13 qubits 33 -> 0.7 ms.
#include <math.h>
#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <numeric>
#include <vector>

#include "common.cuh"
#include "fusion.h"
#include "tile_regs.cuh"
#include "widen.cuh"

namespace qcs {

struct BInst {
  int n;
  int stage0;
  int nstages;
  int group;  // times it is queued: CTAs that start on it
  int tickets;  // of a stage, at most
};

struct BStage {
  int group0;
  int ngroups;
  int nt;             // tile qubits (local bits)
  int pad;
  signed char q[24];  // local bit m -> global qubit (ascending)
};

// A stage's gates run in groups of consecutive gates on a few tile bits: one
// pass over shared memory applies a group, each thread holding the amplitudes
// of one setting of the other bits in registers.  Register bit j is tile bit
// q[j]; bits the gates leave free are filled with others.  Register bit 0 (the
// pair bit, tile_regs.cuh) is the one with the fewest 2x2 gates.
// CTAs of 256 threads hold 2^5 amplitudes a thread: against 2^4 that halves
// the dispatch per amplitude and takes a tenth of the passes away (304
// instances of 18 qubits, 10 layers: 13.7 -> 12.9 ms; 608 of 13 qubits 0.62 ->
// 0.50).  Larger CTAs have no registers for it (at 1024 threads 0.84 -> 1.28).
// The order of the gates comes from a greedy partition into groups on at most
// kGroupQ qubits, and one-qubit gates fold into one 2x2 within those.
constexpr int kGroupQ = 4;
constexpr int kMaxRegQ = 5;
constexpr int reg_q(int threads) { return threads == 256 ? 5 : 4; }
struct __align__(16) BGroup {
  int gate0;
  int ngates;
  unsigned char q[kMaxRegQ];    // tile bit of register bit j
  unsigned char asc[kMaxRegQ];  // the same tile bits, ascending
  unsigned char pad[6];
};

// A planned gate.  p: a 2x2's four complex entries (dense), its two diagonal
// ones (diag) or the phase.
enum { BG_DENSE = 0, BG_EXCH = 8, BG_DIAG = 16, BG_PHASE = 24 };  // + register bit
struct __align__(16) BGate {
  float p[8];
  int op;    // BG_* + target register bit (BG_PHASE: no addition)
  int cond;  // register bits that must be set (exchange: the control or 0)
  int pad[2];
};

struct BatchTune {
  int threads;      // 256, 512 or 1024
  int tile_q;       // 12, 13 or 14
  int ctas_per_sm;  // 1, 2 or 4 (as many run as shared memory and registers allow)
  int order;        // 0: largest first, 1: given order
  int split_q;      // instances above split_q qubits are queued for 2^(n - split_q) CTAs
};

}  // namespace qcs

struct qcs_cuda_batch {
  int count;
  int shots;
  unsigned long long seed;
  int max_n;
  std::vector<int> nq;            // qubits per instance
  std::vector<qcs_cuda_op> ops;   // all ops, instance after instance
  std::vector<int> op_off;        // count + 1
  // plan (for the current tile size)
  std::vector<qcs::BInst> insts;
  std::vector<qcs::BStage> stages;
  std::vector<qcs::BGroup> groups;
  // planned gates in group order: gate i is the product of the ops
  // fold_ops[fold_off[i] .. fold_off[i+1]) (one-qubit gates on one qubit with
  // nothing else on that qubit between them fold into one 2x2)
  std::vector<int> fold_off;
  std::vector<int> fold_ops;
  std::vector<int> gate_tc;       // its group-local target | control << 8 (control 0xFF: none)
  std::vector<int> order;         // instance order
  std::vector<int2> items;        // (instance, member) in queue order, then those in slots
  int n_items;                    // of the queue
  qcs::BatchTune tune;
  int planned_tile_q, planned_regs;
  // device
  cudaStream_t stream;
  qcs::DeviceInfo dev;
  qcs::BInst *d_insts;
  qcs::BStage *d_stages;
  qcs::BGroup *d_groups;
  qcs::BGate *d_gates;
  qcs::BGate *h_gates;  // pinned; the graph's upload node reads it
  int2 *d_items;
  // zeroed by every launch: the queue's head, the slots in use, the shared
  // instances' tickets
  char *d_counters;
  size_t counter_bytes;
  double *d_z;
  double *h_z;          // pinned
  qcs::i64 *d_samples;
  qcs::i64 *h_samples;  // pinned
  float2 *d_slots;      // as many global slots as CTAs, for instances above tile_q
  double *d_sums;       // their read-outs' block sums
  int *d_err;
  long long wait_captured;  // wait limit the captured graph's kernel carries
  size_t slot_amps;
  int grid;
  size_t cap_gates, cap_stages;
  cudaGraphExec_t graph;
  float last_ms;
};

namespace qcs {

constexpr int kMassTile = 4096;  // sampling tile (amplitudes)

__device__ __forceinline__ u64 splitmix64(u64 x) {
  x += 0x9E3779B97F4A7C15ULL;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ULL;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBULL;
  return x ^ (x >> 31);
}

// Uniform draw in [0, 1) for (seed, instance, shot), 53 random bits.
__host__ __device__ inline double shot_draw(u64 seed, u64 inst, u64 shot) {
  u64 x = seed ^ (inst * 0xD1B54A32D192ED03ULL) ^ (shot * 0x8CB92BA72F3D8DD7ULL);
  x += 0x9E3779B97F4A7C15ULL;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ULL;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBULL;
  x ^= x >> 31;
  return (double)(x >> 11) * (1.0 / 9007199254740992.0);
}

__device__ __forceinline__ double bwarp_sum(double x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

template <int T>
__device__ double block_sum(double v, double *red) {
  v = bwarp_sum(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  double r = 0.0;
  if (w == 0) {
    r = l < T / 32 ? red[l] : 0.0;
    r = bwarp_sum(r);
  }
  return r;  // valid in thread 0
}

// The groups of a stage and their gates, as far as they fit: a window copied to
// shared memory, where the tiles that stream through L1 do not push them out.
// A stage that fits whole is copied once for all its tiles; a longer one moves
// the window along.  (Kept there as packed operands, twelve of them, the
// constants of a gate did not fit the registers any more: 12.8 -> 14.0 ms for
// 304 instances of 18 qubits.)
constexpr int kWinGroups = 64, kWinGates = 256;
struct BWindow {
  BGate gate[kWinGates];
  BGroup group[kWinGroups];
};

// X on register bit TB under the control mask `cond` (one bit, or none).
template <int TB, int RB>
__device__ __forceinline__ void batch_exchange(RegsF32<RB> &a, int cond) {
  each<RB>([&](auto cc) {
    constexpr int CB = decltype(cc)::value;
    if constexpr (CB != TB)
      if (cond == 1 << CB) a.template exchange<TB, CB>();
  });
  if (cond == 0) a.template exchange<TB, -1>();
}

template <int RB>
__device__ __forceinline__ void batch_gate(RegsF32<RB> &a, const BGate &g) {
  const float4 x = *reinterpret_cast<const float4 *>(g.p);
  const float4 y = *reinterpret_cast<const float4 *>(g.p + 4);
  const float k[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
  const int op = g.op;
  auto target = [&](auto &&f) {  // f(target bit), as a constant
    if (RB > 4 && (op & 4)) f(std::integral_constant<int, RB - 1>());
    else if (op & 2) {
      if (op & 1) f(std::integral_constant<int, 3>());
      else f(std::integral_constant<int, 2>());
    } else {
      if (op & 1) f(std::integral_constant<int, 1>());
      else f(std::integral_constant<int, 0>());
    }
  };
  if (op < BG_EXCH) target([&](auto tb) { a.template dense<decltype(tb)::value>(k); });
  else if (op < BG_DIAG) target([&](auto tb) { batch_exchange<decltype(tb)::value>(a, g.cond); });
  else if (op < BG_PHASE) target([&](auto tb) { a.template diag<decltype(tb)::value>(k); });
  else a.phase_where(k, g.cond);
}

// Apply one group to a tile of 2^nt amplitudes (nt >= RB) in shared memory.
template <int T, int RB>
__device__ __forceinline__ void smem_group(float *S, int nt, const BGroup &G, const BGate *gates) {
  constexpr int N = 1 << RB;
  const int L = 1 << nt, np = L >> RB;
  const float2 kind = {};
  int m[RB];
#pragma unroll
  for (int j = 0; j < RB; j++) m[j] = tile_pos(1 << G.q[j], kind);
  for (int p = threadIdx.x; p < np; p += T) {
    int l = p;  // a zero inserted at each register bit, ascending
#pragma unroll
    for (int j = 0; j < RB; j++)
      l = ((l >> G.asc[j]) << (G.asc[j] + 1)) | (l & ((1 << G.asc[j]) - 1));
    int at = tile_pos(l, kind);
    auto place = [&](int (&pos)[N]) {
      int lo[4], hi[N / 4];
#pragma unroll
      for (int k = 0; k < 4; k++) lo[k] = at ^ ((k & 1) ? m[0] : 0) ^ ((k & 2) ? m[1] : 0);
#pragma unroll
      for (int k = 0; k < N / 4; k++)
        hi[k] = ((k & 1) ? m[2] : 0) ^ ((k & 2) ? m[3] : 0) ^ ((k & 4) ? m[RB - 1] : 0);
#pragma unroll
      for (int e = 0; e < N; e++) pos[e] = lo[e & 3] ^ hi[e >> 2];
    };
    RegsF32<RB> a;
    {
      int pos[N];
      place(pos);
      a.load(S, L, pos);
    }
    for (int gi = 0; gi < G.ngates; gi++) batch_gate(a, gates[gi]);
    asm volatile("" : "+r"(at));  // the positions are formed anew, not kept
    {
      int pos[N];
      place(pos);
      a.store(S, L, pos);
    }
  }
}

template <int T>
__device__ __forceinline__ void run_groups(float *S, const BStage &st, BWindow &W, int &w0, int &w1,
                                           const BGroup *groups, const BGate *gates) {
  const int end = st.group0 + st.ngroups;
  for (int gi = st.group0; gi < end; gi++) {
    if (gi < w0 || gi >= w1) {  // (the same decision in every thread)
      __syncthreads();
      const int n = end - gi < kWinGroups ? end - gi : kWinGroups;
      for (int e = threadIdx.x; e < n; e += T) W.group[e] = groups[gi + e];
      __syncthreads();
      const int g0 = W.group[0].gate0;
      int fit = 1;  // a group has at most kWinGates gates
      while (fit < n && W.group[fit].gate0 + W.group[fit].ngates - g0 <= kWinGates) fit++;
      const int count = W.group[fit - 1].gate0 + W.group[fit - 1].ngates - g0;
      const float4 *src = reinterpret_cast<const float4 *>(gates + g0);
      float4 *dst = reinterpret_cast<float4 *>(W.gate);
      for (int e = threadIdx.x; e < 3 * count; e += T) dst[e] = src[e];
      w0 = gi;
      w1 = gi + fit;
      __syncthreads();
    }
    const BGroup &G = W.group[gi - w0];
    smem_group<T, reg_q(T)>(S, st.nt, G, W.gate + (G.gate0 - W.group[0].gate0));
    __syncthreads();
  }
}

// ---- read-outs ----------------------------------------------------------
// <Z_0> and the sampling tiles' masses are FP64 sums of FP32 squares; inside a
// tile a shot follows running sums of exact squares in FP64.  All of it is
// bound by the FP64 pipe, so floats are widened with integer operations
// (widen.cuh), the squares go straight into the sums by FMA, and no amplitude is summed twice: every block of 32 or
// more amplitudes is summed once, by whichever CTA is free, and a shot (a
// thread) searches the running sums and then one block.  Against a scan of the
// shot's tile, 4096 amplitudes or more, by a warp of the instance's one CTA: 384
// instances of 12-16 qubits 10.5 -> 1.6 ms, 96 of 10-20 11.5 -> 2.9, 384 of
// 10-22 72 -> 63, 8 of 18-22 12.4 -> 4.1 (with more tickets a stage).

__device__ __forceinline__ float prob32(float2 a) { return a.x * a.x + a.y * a.y; }
__device__ __forceinline__ bool nonzero(float2 a) { return a.x != 0.f || a.y != 0.f; }

// cum[k] = c + the squares of a[0 .. k].
template <bool PLAIN>
__device__ __forceinline__ void running8(const float2 (&a)[8], double c, double (&cum)[8]) {
#pragma unroll
  for (int k = 0; k < 8; k++) {
    const double x = to64<PLAIN>(a[k].x), y = to64<PLAIN>(a[k].y);
    c = fma(x, x, c);
    c = fma(y, y, c);
    cum[k] = c;
  }
}

// The sums of a block: FP32 squares of its even and odd amplitudes, and FP64 squares.
struct BlockSums {
  double even = 0.0, odd = 0.0, exact = 0.0;
  template <bool PLAIN>
  __device__ __forceinline__ void add(const float2 (&a)[8], const float (&p)[8]) {
#pragma unroll
    for (int k = 0; k < 8; k += 2) {
      even += to64<PLAIN>(p[k]);
      odd += to64<PLAIN>(p[k + 1]);
    }
    double c[8];
    running8<PLAIN>(a, exact, c);
    exact = c[7];
  }
  __device__ __forceinline__ void add(const float2 (&a)[8]) {  // a[0]: an even amplitude
    float p[8];
    PlainTest t;
#pragma unroll
    for (int k = 0; k < 8; k++) {
      p[k] = prob32(a[k]);
      t.see(p[k]);
      t.see(a[k].x);
      t.see(a[k].y);
    }
    if (t.plain()) add<true>(a, p);
    else add<false>(a, p);
  }
};

// Exclusive prefix of x[0 .. m) in shared memory, the total at x[m], by one
// warp: each lane sums its run of entries, the warp scans the runs.
__device__ void warp_prefix(double *x, int m) {
  const int lane = threadIdx.x & 31;
  const int per = (m + 31) / 32, i0 = lane * per < m ? lane * per : m;
  const int i1 = i0 + per < m ? i0 + per : m;
  double s = 0.0;
  for (int i = i0; i < i1; i++) s += x[i];
  double incl = s;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const double y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  double run = __shfl_up_sync(0xffffffffu, incl, 1);
  if (lane == 0) run = 0.0;
  __syncwarp();
  for (int i = i0; i < i1; i++) {
    const double v = x[i];
    x[i] = run;
    run += v;
  }
  const double total = __shfl_sync(0xffffffffu, incl, 31);
  if (lane == 0) x[m] = total;
}

constexpr int kBlock = 32;        // amplitudes of a block in a slot, at least
constexpr int kMaxBlocks = 8192;  // blocks of an instance
constexpr int kMaxTiles = 1024;   // sampling tiles of an instance

struct ReadShape {
  i64 block, tile;  // amplitudes
  int n_blocks, n_tiles, per;  // per: blocks of a tile
};
__host__ __device__ inline ReadShape read_shape(i64 size, int block = kBlock) {
  ReadShape r;
  r.block = size / kMaxBlocks > block ? size / kMaxBlocks : block;
  r.tile = size / kMaxTiles > kMassTile ? size / kMaxTiles : kMassTile;
  if (r.tile > size) r.tile = size;
  if (r.block > size) r.block = size;
  r.n_blocks = (int)(size / r.block);
  r.n_tiles = (int)(size / r.tile);
  r.per = (int)(r.tile / r.block);
  return r;
}

// From the blocks' sums: prefix[0 .. n_tiles], the tiles' running masses, and
// incl[b], the running sum of exact squares within b's tile (incl may be
// `exact`).  1 to 32 lanes a tile, a run of its blocks each.  GLOBAL: the sums
// are in global memory, written by several CTAs.
template <int T, bool GLOBAL>
__device__ void running_sums(const ReadShape &R, const double *mass, const double *exact,
                             double *incl, double *prefix) {
  const int g = R.per < 8 ? 1 : R.per / 8 < 32 ? R.per / 8 : 32, run = R.per / g;
  for (int u0 = 0; u0 < R.n_tiles * g; u0 += T) {  // full warps: they shuffle
    const int u = u0 + threadIdx.x;
    const bool valid = u < R.n_tiles * g;
    const int j = u & (g - 1), b0 = u * run;
    double m = 0.0, s = 0.0;
    if (valid)
      for (int k = 0; k < run; k++) {
        m += GLOBAL ? __ldcg(mass + b0 + k) : mass[b0 + k];
        s += GLOBAL ? __ldcg(exact + b0 + k) : exact[b0 + k];
      }
    double up = s;
    for (int o = 1; o < g; o <<= 1) {
      m += __shfl_xor_sync(0xffffffffu, m, o);
      const double y = __shfl_up_sync(0xffffffffu, up, o);
      if (j >= o) up += y;
    }
    double before = __shfl_up_sync(0xffffffffu, up, 1);
    if (j == 0) before = 0.0;
    if (!valid) continue;
    if (j == 0) prefix[u / g] = m;
    for (int k = 0; k < run; k++) {
      before += GLOBAL ? __ldcg(exact + b0 + k) : exact[b0 + k];
      incl[b0 + k] = before;
    }
  }
  __syncthreads();
  if (threadIdx.x < 32) warp_prefix(prefix, R.n_tiles);
  __syncthreads();
}

// The shots, a thread each: its tile and its block by binary search over
// running sums, then the block's amplitudes; load8(i, a) gives amplitudes
// i .. i+7 (those from the instance's size on are 0).
template <int T, class Load8>
__device__ __forceinline__ void pick_shots(const ReadShape &R, const double *prefix,
                                           const double *incl, int shots, u64 seed, int inst,
                                           i64 *out, const Load8 &load8) {
  for (int s = threadIdx.x; s < shots; s += T) {
    const double r = shot_draw(seed, (u64)inst, (u64)s);
    i64 result = -1;
    if (r < prefix[R.n_tiles]) {
      int t = 0, last = R.n_tiles - 1;
      while (t < last) {
        const int mid = (t + last) >> 1;
        if (r < prefix[mid + 1]) last = mid;
        else t = mid + 1;
      }
      const double base = prefix[t];
      const int first = t * R.per, end = first + R.per;
      int lo = first, hi = end;  // the first block with r < base + its running sum
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (r < base + incl[mid]) hi = mid;
        else lo = mid + 1;
      }
      i64 from = t * R.tile, to = from + R.tile;  // where the last nonzero one is taken
      if (lo < end) {
        double cum = lo > first ? base + incl[lo - 1] : base;
        from = lo * R.block;
        to = from + R.block;
        for (i64 i = from; i < to && result < 0; i += 8) {
          float2 a[8];
          load8(i, a);
          PlainTest test;
#pragma unroll
          for (int k = 0; k < 8; k++) {
            test.see(a[k].x);
            test.see(a[k].y);
          }
          double c[8];
          if (test.plain()) running8<true>(a, cum, c);
          else running8<false>(a, cum, c);
          cum = c[7];
          if (!(r < cum)) continue;
#pragma unroll
          for (int k = 7; k >= 0; k--)
            if (nonzero(a[k]) && r < c[k]) result = i + k;
        }
      }
      if (result < 0) {
        result = from;
        for (i64 i = (to - 1) & ~(i64)7; i >= from && result == from; i -= 8) {
          float2 a[8];
          load8(i, a);
#pragma unroll
          for (int k = 0; k < 8; k++)
            if (nonzero(a[k])) result = i + k;
        }
      }
    }
    out[s] = result;
  }
}

// Read-out of an instance that lives in shared memory (L = 2^n amplitudes of
// a tile of Lt; those from L on are 0).  Returns <Z_0> in thread 0.
// A block's sums are chains of FP64 additions in one thread, so small instances
// have blocks of fewer than 32 amplitudes, up to 256 of them (20000 of 5 qubits, 20
// gates, 16 shots: 1144 -> 775 us).
// scratch: 5 + 2 * (L / 32 or 256) doubles.
template <int T>
__device__ double resident_readout(const float *S, int L, int Lt, double *scratch, double *red,
                                   int shots, u64 seed, int inst, i64 *out) {
  const float2 kind = {};
  const ReadShape R = read_shape(L, L >= 256 * kBlock ? kBlock : L >= 4096 ? L / 256 : 8);
  double *prefix = scratch, *exact = scratch + 5, *mass = exact + R.n_blocks;
  auto load8 = [&](i64 i, float2 (&a)[8]) {
#pragma unroll
    for (int k = 0; k < 8; k++) a[k] = tile_get(S, Lt, tile_pos((int)i + k, kind));
  };
  double z = 0.0;
  for (int b = threadIdx.x; b < R.n_blocks; b += T) {
    BlockSums sums;
    for (int k = 0; k < (int)R.block; k += 8) {
      float2 a[8];
      load8(b * R.block + k, a);
      sums.add(a);
    }
    exact[b] = sums.exact;
    mass[b] = sums.even + sums.odd;
    z += sums.even - sums.odd;
  }
  z = block_sum<T>(z, red);
  if (shots == 0) return z;
  __syncthreads();
  running_sums<T, false>(R, mass, exact, exact, prefix);
  pick_shots<T>(R, prefix, exact, shots, seed, inst, out, load8);
  return z;
}

// Read-out of an instance in its global slot.  The block sums are tickets:
// part `part` of `parts`, four lanes a block; sums: mass, even - odd and exact
// square sum of each block.
template <int T>
__device__ void slot_sums(const float2 *slot, i64 size, int part, int parts, double *sums) {
  const ReadShape R = read_shape(size);
  const int n = R.n_blocks / parts;  // at least 2^tile_q / 32
  const int j = threadIdx.x & 3;
  for (int b0 = 0; b0 < n; b0 += T / 4) {  // full warps: they shuffle
    const int b = part * n + b0 + threadIdx.x / 4;
    const bool valid = b0 + threadIdx.x / 4 < n;
    BlockSums s;
    if (valid) {
      const float4 *v = reinterpret_cast<const float4 *>(slot + b * R.block) + j;
      for (i64 i = 0; i < R.block; i += 32, v += 16) {
        float2 a[8];
#pragma unroll
        for (int k = 0; k < 4; k++) {
          const float4 x = __ldcg(v + 4 * k);
          a[2 * k] = make_float2(x.x, x.y);
          a[2 * k + 1] = make_float2(x.z, x.w);
        }
        s.add(a);
      }
    }
    double mass = s.even + s.odd, diff = s.even - s.odd;
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) {
      mass += __shfl_xor_sync(0xffffffffu, mass, o);
      diff += __shfl_xor_sync(0xffffffffu, diff, o);
      s.exact += __shfl_xor_sync(0xffffffffu, s.exact, o);
    }
    if (valid && j < 3) sums[(i64)j * R.n_blocks + b] = j == 0 ? mass : j == 1 ? diff : s.exact;
  }
}

// The rest, once all sums are there.  room: space for `room_blocks` doubles in
// shared memory.  Returns <Z_0> in thread 0.
template <int T>
__device__ double slot_readout(const float2 *slot, i64 size, double *sums, double *room,
                               int room_blocks, double *prefix, double *red, int shots, u64 seed,
                               int inst, i64 *out) {
  const ReadShape R = read_shape(size);
  const double *mass = sums, *diff = sums + R.n_blocks;
  double *exact = sums + 2 * (i64)R.n_blocks;
  double *incl = R.n_blocks <= room_blocks ? room : exact;
  double z = 0.0;
  for (int b = threadIdx.x; b < R.n_blocks; b += T) z += __ldcg(diff + b);
  z = block_sum<T>(z, red);
  __syncthreads();
  running_sums<T, true>(R, mass, exact, incl, prefix);
  pick_shots<T>(R, prefix, incl, shots, seed, inst, out, [&](i64 i, float2 (&a)[8]) {
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const float4 x = __ldcg(reinterpret_cast<const float4 *>(slot + i) + k);
      a[2 * k] = make_float2(x.x, x.y);
      a[2 * k + 1] = make_float2(x.z, x.w);
    }
  });
  return z;
}

// Thread 0 waits until *cnt >= target, at most `limit` clock cycles; false
// on timeout or abort.
__device__ bool wait_count(const int *cnt, int target, int *err, int where, long long limit) {
  const long long t0 = clock64();
  while (*(volatile const int *)cnt < target) {
    if (*(volatile const int *)err) return false;
    if (clock64() - t0 > limit) {
      atomicCAS(err, 0, where);
      return false;
    }
    __nanosleep(200);
  }
  __threadfence();
  return true;
}

// Per instance in a global slot, zero before a launch.
struct BShare {
  int next;  // the next ticket
  int done;  // tickets whose tiles are written
  int slot;  // 1 + the slot that holds the amplitudes
  int at_it; // CTAs that take its tickets
};

// How an instance in a global slot is shared.  Its work is a line of tickets,
// `chunk` tiles of one stage each, stage after stage; any CTA takes the next
// ticket, waits until every ticket of the earlier stages is done, does its
// tiles and counts it done; whoever counts the last one reads the instance
// out.  A CTA waits only for lower tickets, each in the hands of a CTA that
// works on it, so nothing depends on which CTAs run at the same time or on
// when they join: an instance is queued `group` times, and CTAs that find the
// queue empty join the instances that still have tickets.
// Fixed members that met after every stage idled until the last of them had
// come free, and left the rest of the GPU idle at the end of the batch: 96
// instances of 10-20 qubits 34 -> 11.5 ms, 24 of 12-22 36 -> 16.3, 8 of 18-22
// 29 -> 12.4, 384 of 10-22 85 -> 72.
struct BTickets {
  int chunk, per_stage, total;
};
__device__ __forceinline__ BTickets batch_tickets(const BInst &I, int tile_q) {
  const int n_tiles = 1 << (I.n - tile_q);
  BTickets k;
  k.chunk = n_tiles > I.tickets ? n_tiles / I.tickets : 1;
  k.per_stage = n_tiles / k.chunk;
  k.total = k.per_stage * (I.nstages + 1);  // the read-out's sums are the last stage
  return k;
}

template <int T>
__global__ void __launch_bounds__(T, T == 256 ? 2 : 1)
    k_batch(const BInst *insts, const BStage *stages, const BGroup *groups, const BGate *gates,
            const int2 *items, int n_items, int n_slot, int shots, u64 seed, int tile_q, float2 *slots,
            i64 slot_amps, double *slot_sum, i64 sums_of_slot, int *queue, BShare *share, int *slot_busy, int *err, double *z_out,
            i64 *samples_out, long long wait) {
  QCS_REGS_F32_DECLARE(1 << (reg_q(T) - 1));
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float *S = reinterpret_cast<float *>(smem_raw);                      // 2^tile_q amplitudes
  BWindow &W = *reinterpret_cast<BWindow *>(S + (2 << tile_q));
  double *scratch = reinterpret_cast<double *>(&W + 1);  // of the read-outs
  __shared__ double red[T / 32];
  __shared__ int s_pick, s_ticket, s_slot, s_ok;
  __shared__ u64 s_best;
  // of the stage: a thread's accesses to a tile, and the tile's base by
  // nibbles of its number
  __shared__ i64 step_off[64], nib[4][16];
  const float2 kind = {};

  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) s_pick = atomicAdd(queue, 1);
    __syncthreads();
    int inst;
    const bool joined = s_pick >= n_items;
    if (!joined) {
      inst = items[s_pick].x;
    } else if (n_slot == 0) {
      break;
    } else {
      // the queue is empty: join the instance with the most tiles left per CTA
      // at it (those in slots are listed after the queue).  A CTA that joins
      // changes at_it, so of those that chose the same instance one gets it and
      // the others look again.
      // (The upper half of the grid, whose CTAs lie beside one of the lower half on
      // an SM, lets that go first: one instance of 16 qubits, eight CTAs, takes 388
      // us where they have eight SMs and 535 where two share one.)
      if (2 * blockIdx.x >= gridDim.x) __nanosleep(4000);
      do {
        __syncthreads();
        if (threadIdx.x == 0) s_best = 0;
        __syncthreads();
        for (int e = threadIdx.x; e < n_slot; e += T) {
          const int2 it = items[n_items + e];
          if (it.x >= 1 << 24) continue;
          const BInst J = insts[it.x];
          const BTickets k = batch_tickets(J, tile_q);
          const int left = k.total - *(volatile int *)&share[it.x].next;
          const int at_it = *(volatile int *)&share[it.x].at_it;
          if (left <= 0 || at_it >= k.per_stage) continue;
          const int each = min(left * k.chunk / (at_it + 1) + 1, 0xffffff);
          atomicMax(&s_best, (u64)each << 40 | (u64)at_it << 24 | it.x);
        }
        __syncthreads();
        inst = s_best ? (int)(s_best & 0xffffff) : -1;
        if (threadIdx.x == 0 && inst >= 0) {
          const int at_it = (int)(s_best >> 24) & 0xffff;
          s_ok = atomicCAS(&share[inst].at_it, at_it, at_it + 1) == at_it;
        }
        __syncthreads();
      } while (inst >= 0 && !s_ok);
      if (inst < 0) break;
    }
    const BInst I = insts[inst];
    const i64 size = 1LL << I.n;
    double z = 0.0;
    int w0 = 0, w1 = 0;  // groups in the window
    i64 *out = samples_out + (i64)inst * shots;
    if (I.n <= tile_q) {
      // ---- shared-memory resident instance (a tile of at least 2^kMaxRegQ) ----
      const BStage st = stages[I.stage0];
      const int Lt = 1 << st.nt;
      for (int i = threadIdx.x; i < 2 * Lt; i += T) S[i] = i == 0 ? 1.f : 0.f;  // position 0
      __syncthreads();
      run_groups<T>(S, st, W, w0, w1, groups, gates);
      z = resident_readout<T>(S, (int)size, Lt, scratch, red, shots, seed, inst, out);
      if (threadIdx.x == 0) z_out[inst] = z;
      continue;
    }
    // ---- global-slot instance, run in stages ----
    const BTickets K = batch_tickets(I, tile_q);
    BShare *sh = share + inst;
    BStage st;
    int stage = -1;
    // of the stage, for this thread (see below)
    i64 toff = 0;
    const int i0 = 2 * threadIdx.x;  // its first amplitude
    const int tpos = tile_pos(i0, kind);
    const int L = 1 << tile_q;
    const int steps = L / 2 > T ? L / 2 / T : 1;
    const bool active = i0 < L;
    // The next ticket is taken before the tiles of this one, so that its first
    // tile is known early enough to be fetched.
    if (threadIdx.x == 0) {
      if (!joined) atomicAdd(&sh->at_it, 1);
      s_ticket = atomicAdd(&sh->next, 1);
    }
    __syncthreads();
    int ticket = s_ticket;
    float2 *slot = nullptr;
    while (ticket < K.total) {
      const int si = ticket / K.per_stage;
      __syncthreads();
      if (threadIdx.x == 0) {
        s_ok = 1;
        if (ticket == 0) {  // this CTA opens the instance: a free slot
          // (at most one instance is open per CTA of the grid)
          int k = blockIdx.x, tries = 0;
          while (atomicCAS(&slot_busy[k], 0, 1) != 0 && tries < (1 << 16)) {
            k = k + 1 < (int)gridDim.x ? k + 1 : 0;
            tries++;
          }
          if (tries < (1 << 16)) {
            atomicExch(&sh->slot, k + 1);
          } else {  // after a wait that ran out: its instances keep their slots
            atomicCAS(err, 0, 3);
            s_ok = 0;
          }
        } else if (slot == nullptr) {
          s_ok = wait_count(&sh->slot, 1, err, 1, wait) ? 1 : 0;
        }
        if (s_ok && si != stage && si > 0)
          s_ok = wait_count(&sh->done, si * K.per_stage, err, 2, wait) ? 1 : 0;
        s_slot = *(volatile int *)&sh->slot - 1;
        s_ticket = atomicAdd(&sh->next, 1);
      }
      __syncthreads();
      if (!s_ok) return;
      slot = slots + (i64)s_slot * slot_amps;
      double *sums = slot_sum + (i64)s_slot * sums_of_slot;
      const int next = s_ticket;
      if (si == I.nstages) {
        slot_sums<T>(slot, size, ticket - si * K.per_stage, K.per_stage, sums);
      } else if (si != stage) {
        stage = si;
        st = stages[I.stage0 + si];
        // A thread moves units of two amplitudes (16 bytes; tile bit 0 is
        // qubit 0): unit t + k T, whose offset is that of t plus that of k T.
        for (int e = threadIdx.x; e < 64 + 64; e += T) {
          if (e < 64) {
            i64 o = 0;
            for (int m = 0; m < tile_q; m++)
              if (((e * T * 2) >> m) & 1) o |= 1LL << st.q[m];
            step_off[e] = o;
          } else {  // qubits outside the tile, ascending: the tile number's bits
            const int k = (e - 64) >> 4, v = (e - 64) & 15;
            i64 o = 0;
            int j = 0, in = 0;
            for (int q = 0; q < I.n; q++) {
              if (in < tile_q && st.q[in] == q) {
                in++;
                continue;
              }
              if ((j >> 2) == k && ((v >> (j & 3)) & 1)) o |= 1LL << q;
              j++;
            }
            nib[k][v] = o;
          }
        }
        toff = 0;
        for (int m = 1; m < tile_q; m++)
          if ((i0 >> m) & 1) toff |= 1LL << st.q[m];
        __syncthreads();
      }
      auto tile_at = [&](int tt) {  // this thread's first unit of a tile
        return slot + nib[0][tt & 15] + nib[1][(tt >> 4) & 15] + nib[2][(tt >> 8) & 15] +
               nib[3][(tt >> 12) & 15] + toff;
      };
      const int t0 = (ticket - si * K.per_stage) * K.chunk;
      for (int tt = t0; si < I.nstages && tt < t0 + K.chunk; tt++) {
        float2 *vt = tile_at(tt);
        if (si == 0) {  // |0...0>
          for (int i = threadIdx.x; i < 2 * L; i += T) S[i] = tt == 0 && i == 0 ? 1.f : 0.f;
        } else if (active) {
          for (int k0 = 0; k0 < steps; k0 += 4) {
            float4 x[4];
#pragma unroll
            for (int k = 0; k < 4; k++)
              if (k0 + k < steps)
                x[k] = __ldcg(reinterpret_cast<const float4 *>(vt + step_off[k0 + k]));
#pragma unroll
            for (int k = 0; k < 4; k++) {
              if (k0 + k >= steps) break;
              const int at = tpos ^ tile_pos((k0 + k) * T * 2, kind);
              tile_put(S, L, at, make_float2(x[k].x, x[k].y));
              tile_put(S, L, at ^ 1, make_float2(x[k].z, x[k].w));
            }
          }
        }
        __syncthreads();
        const int after = tt + 1 < t0 + K.chunk ? tt + 1
                          : next / K.per_stage == si ? (next - si * K.per_stage) * K.chunk : -1;
        if (si > 0 && active && after >= 0) {  // the next tile, towards L2
          const float2 *vn = tile_at(after);
          for (int k = 0; k < steps; k++)
            asm volatile("prefetch.global.L2 [%0];" ::"l"(vn + step_off[k]));
        }
        run_groups<T>(S, st, W, w0, w1, groups, gates);
        if (active) {
          for (int k = 0; k < steps; k++) {
            const int at = tpos ^ tile_pos(k * T * 2, kind);
            const float2 x = tile_get(S, L, at), y = tile_get(S, L, at ^ 1);
            *reinterpret_cast<float4 *>(vt + step_off[k]) = make_float4(x.x, x.y, y.x, y.y);
          }
        }
        __syncthreads();
      }
      __threadfence();  // each thread's slot writes, before the count
      __syncthreads();
      if (threadIdx.x == 0) {
        __threadfence();
        s_ok = atomicAdd(&sh->done, 1) == K.total - 1;
        __threadfence();
      }
      __syncthreads();
      if (s_ok) {  // the last one: the whole state is written
        z = slot_readout<T>(slot, size, sums, reinterpret_cast<double *>(S), L, scratch, red, shots,
                            seed, inst, out);
        if (threadIdx.x == 0) z_out[inst] = z;
        __syncthreads();
        if (threadIdx.x == 0) atomicExch(&slot_busy[s_slot], 0);
      }
      ticket = next;
    }
    if (threadIdx.x == 0) atomicSub(&sh->at_it, 1);
  }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------

// The gates of one stage (op indices in order) on tile qubits tq (ascending):
// a greedy partition into groups on at most kGroupQ qubits (commuting only past
// gates on disjoint qubits) gives their order and the one-qubit gates that
// fold into one 2x2; the sequence is then cut, in order, into register groups
// on at most `regs` tile bits (and of as many gates as the window holds).
static void plan_groups(qcs_cuda_batch *b, const std::vector<int> &stage_ops, int n,
                        const std::vector<int> &tq, int regs, BStage &st) {
  st.group0 = (int)b->groups.size();
  std::vector<qcs_cuda_op> sub(stage_ops.size());
  for (size_t j = 0; j < stage_ops.size(); j++) sub[j] = b->ops[stage_ops[j]];
  PartitionOptions po;
  po.kmax = kGroupQ;
  po.cost = nullptr;
  po.cost_ctx = nullptr;
  std::vector<PlanItem> items = partition(sub.data(), (int)sub.size(), n, po);
  auto tile_bit = [&](int q) {
    for (size_t m = 0; m < tq.size(); m++)
      if (tq[m] == q) return (int)m;
    return -1;
  };
  struct Planned {
    std::vector<int> ops;  // that it folds
    int t, c;              // tile bits (c: -1 for one-qubit gates)
  };
  std::vector<Planned> seq;
  for (const PlanItem &it : items) {
    // pending[m]: the one-qubit gate on tile bit m that later one-qubit gates
    // on m fold into, -1 after a two-qubit gate touched m
    std::vector<int> pending(st.nt, -1);
    for (int g : it.gates) {
      const qcs_cuda_op &o = sub[g];
      const int t = tile_bit(o.target);
      if (gate_is_controlled(o.kind)) {
        const int c = tile_bit(o.control);
        pending[t] = pending[c] = -1;
        seq.push_back({{stage_ops[g]}, t, c});
      } else if (pending[t] >= 0) {
        seq[pending[t]].ops.push_back(stage_ops[g]);
      } else {
        pending[t] = (int)seq.size();
        seq.push_back({{stage_ops[g]}, t, -1});
      }
    }
  }
  for (size_t first = 0; first < seq.size();) {
    std::vector<int> bits, uses(st.nt, 0);
    size_t last = first;
    for (; last < seq.size(); last++) {
      const Planned &g = seq[last];
      std::vector<int> more;
      for (int m : {g.t, g.c})
        if (m >= 0 && std::find(bits.begin(), bits.end(), m) == bits.end()) more.push_back(m);
      if (bits.size() + more.size() > (size_t)regs || last - first == kWinGates) break;
      bits.insert(bits.end(), more.begin(), more.end());
      if (g.c < 0) uses[g.t]++;
    }
    // register bits: first tile bits that no gate touches (the highest ones, so
    // that a warp's lanes keep the low ones), then those with the fewest 2x2s
    std::stable_sort(bits.begin(), bits.end(), [&](int x, int y) { return uses[x] < uses[y]; });
    for (int m = st.nt - 1; (int)bits.size() < regs; m--)
      if (std::find(bits.begin(), bits.end(), m) == bits.end()) bits.insert(bits.begin(), m);
    BGroup G;
    memset(&G, 0, sizeof(G));
    G.gate0 = (int)b->gate_tc.size();
    G.ngates = (int)(last - first);
    for (int j = 0; j < regs; j++) G.q[j] = G.asc[j] = (unsigned char)bits[j];
    std::sort(G.asc, G.asc + regs);
    auto reg = [&](int m) { return (int)(std::find(bits.begin(), bits.end(), m) - bits.begin()); };
    for (; first < last; first++) {
      const Planned &g = seq[first];
      b->fold_off.push_back((int)b->fold_ops.size());
      b->fold_ops.insert(b->fold_ops.end(), g.ops.begin(), g.ops.end());
      b->gate_tc.push_back(reg(g.t) | (g.c < 0 ? 0xFF : reg(g.c)) << 8);
    }
    b->groups.push_back(G);
  }
  st.ngroups = (int)b->groups.size() - st.group0;
}

static int batch_plan(qcs_cuda_batch *b, int tile_q, int regs) {
  b->insts.clear();
  b->stages.clear();
  b->groups.clear();
  b->fold_off.clear();
  b->fold_ops.clear();
  b->gate_tc.clear();
  for (int i = 0; i < b->count; i++) {
    BInst I;
    I.n = b->nq[i];
    I.stage0 = (int)b->stages.size();
    I.group = 1;
    const qcs_cuda_op *ops = b->ops.data() + b->op_off[i];
    const int nops = b->op_off[i + 1] - b->op_off[i];
    if (I.n <= tile_q) {
      BStage st;
      memset(&st, 0, sizeof(st));
      st.nt = std::max(I.n, kMaxRegQ);  // qubits a smaller instance lacks stay 0
      std::vector<int> tq(I.n), stage_ops(nops);
      std::iota(tq.begin(), tq.end(), 0);
      std::iota(stage_ops.begin(), stage_ops.end(), b->op_off[i]);
      for (int m = 0; m < I.n; m++) st.q[m] = (signed char)m;
      plan_groups(b, stage_ops, I.n, tq, regs, st);
      b->stages.push_back(st);
      I.nstages = 1;
    } else {
      PartitionOptions po;
      po.kmax = tile_q - 3;
      po.cost = nullptr;
      po.cost_ctx = nullptr;
      std::vector<PlanItem> plan = partition(ops, nops, I.n, po);
      if (plan.empty()) {  // no gates: one empty stage still writes |0...0>
        PlanItem empty;
        empty.kind = 0;
        empty.op = -1;
        plan.push_back(empty);
      }
      for (const PlanItem &it : plan) {
        BStage st;
        memset(&st, 0, sizeof(st));
        std::vector<char> in(I.n, 0);
        for (int q : it.qubits) in[q] = 1;
        int cnt = (int)it.qubits.size();
        for (int q = 0; q < I.n && cnt < tile_q; q++)
          if (!in[q]) {
            in[q] = 1;
            cnt++;
          }
        std::vector<int> tq;
        for (int q = 0; q < I.n; q++)
          if (in[q]) tq.push_back(q);
        st.nt = (int)tq.size();
        for (int m = 0; m < st.nt; m++) st.q[m] = (signed char)tq[m];
        std::vector<int> stage_ops;
        for (int g : it.gates) stage_ops.push_back(b->op_off[i] + g);
        plan_groups(b, stage_ops, I.n, tq, regs, st);
        b->stages.push_back(st);
      }
      I.nstages = (int)plan.size();
    }
    b->insts.push_back(I);
  }
  b->fold_off.push_back((int)b->fold_ops.size());
  b->planned_tile_q = tile_q;
  b->planned_regs = regs;
  return QCS_CUDA_OK;
}

// Gate table from the ops and the current angles (group-local bits): each
// entry is the FP64 product of its folded ops, rounded once to FP32.
static void batch_fill_gates(qcs_cuda_batch *b) {
  const size_t ng = b->gate_tc.size();
  for (size_t gi = 0; gi < ng; gi++) {
    double acc[8] = {1, 0, 0, 0, 0, 0, 1, 0};
    int kind = 0;
    for (int f = b->fold_off[gi]; f < b->fold_off[gi + 1]; f++) {
      const qcs_cuda_op &o = b->ops[b->fold_ops[f]];
      kind = o.kind;
      double m[8], r[8];
      gate_matrix(o.kind, o.angle, m);
      for (int i = 0; i < 2; i++)  // acc := m * acc
        for (int j = 0; j < 2; j++) {
          double re = 0.0, im = 0.0;
          for (int l = 0; l < 2; l++) {
            const double *x = m + 2 * (2 * i + l), *y = acc + 2 * (2 * l + j);
            re += x[0] * y[0] - x[1] * y[1];
            im += x[0] * y[1] + x[1] * y[0];
          }
          r[2 * (2 * i + j)] = re;
          r[2 * (2 * i + j) + 1] = im;
        }
      memcpy(acc, r, sizeof(acc));
    }
    BGate g;
    memset(&g, 0, sizeof(g));
    // exact zeros decide the form: the exchange and diagonal paths give the
    // same numbers as the dense one (the skipped terms are products with 0),
    // and a controlled phase leaves the amplitudes its 1 would multiply
    const bool off0 = acc[2] == 0.0 && acc[3] == 0.0 && acc[4] == 0.0 && acc[5] == 0.0;
    const bool swap = acc[0] == 0.0 && acc[1] == 0.0 && acc[6] == 0.0 && acc[7] == 0.0 &&
                      acc[2] == 1.0 && acc[3] == 0.0 && acc[4] == 1.0 && acc[5] == 0.0;
    const int t = b->gate_tc[gi] & 0xFF;
    const int c = gate_is_controlled(kind) ? (b->gate_tc[gi] >> 8) & 0xFF : -1;
    if (swap) {
      g.op = BG_EXCH + t;
      g.cond = c >= 0 ? 1 << c : 0;
    } else if (c >= 0) {  // CPHASE
      g.op = BG_PHASE;
      g.cond = 1 << t | 1 << c;
      g.p[0] = (float)acc[6];
      g.p[1] = (float)acc[7];
    } else if (off0) {
      g.op = BG_DIAG + t;
      g.p[0] = (float)acc[0];
      g.p[1] = (float)acc[1];
      g.p[2] = (float)acc[6];
      g.p[3] = (float)acc[7];
    } else {
      g.op = BG_DENSE + t;
      for (int e = 0; e < 8; e++) g.p[e] = (float)acc[e];
    }
    b->h_gates[gi] = g;
  }
}

static void batch_free_device(qcs_cuda_batch *b) {
  if (b->graph) cudaGraphExecDestroy(b->graph);
  b->graph = nullptr;
  cudaFree(b->d_insts);
  cudaFree(b->d_stages);
  cudaFree(b->d_groups);
  cudaFree(b->d_gates);
  if (b->h_gates) cudaFreeHost(b->h_gates);
  cudaFree(b->d_items);
  b->d_insts = nullptr;
  b->d_stages = nullptr;
  b->d_groups = nullptr;
  b->d_gates = nullptr;
  b->h_gates = nullptr;
  b->d_items = nullptr;
}

// The tile, the window of gates, then scratch of the read-outs: 1025 prefixes of a slot's sampling
// tiles, or 5 + 2 * 2^tile_q / 32 doubles of a resident instance (5 + 2 * 256 of one
// below 2^13 amplitudes).
static size_t smem_for(int tile_q) {
  const size_t blocks = 5 + 2 * (((size_t)1 << tile_q) / kBlock);
  return ((size_t)8 << tile_q) + sizeof(BWindow) + std::max<size_t>(1025, blocks) * sizeof(double);
}

// CTAs that an SM holds at once: by registers 2 of 256 threads and 1 of 512 or
// 1024, by shared memory fewer.
template <int T>
static int batch_fit_t(int tile_q, int *fit) {
  int rc = check_cuda(cudaFuncSetAttribute(k_batch<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)smem_for(tile_q)),
                      "cudaFuncSetAttribute(batch)");
  if (!rc)
    rc = check_cuda(cudaOccupancyMaxActiveBlocksPerMultiprocessor(fit, k_batch<T>, T,
                                                                  smem_for(tile_q)),
                    "occupancy");
  return rc;
}
static int batch_fit(int threads, int tile_q, int *fit) {
  return threads == 256 ? batch_fit_t<256>(tile_q, fit)
         : threads == 512 ? batch_fit_t<512>(tile_q, fit) : batch_fit_t<1024>(tile_q, fit);
}

// Doubles of a slot's block sums.
static size_t sums_of_slot(const qcs_cuda_batch *b) {
  return 3 * (size_t)read_shape((i64)b->slot_amps).n_blocks;
}

static int batch_upload(qcs_cuda_batch *b) {
  batch_free_device(b);
  int rc = check_cuda(cudaMalloc((void **)&b->d_insts, b->insts.size() * sizeof(BInst)), "cudaMalloc(batch)");
  if (!rc) rc = check_cuda(cudaMalloc((void **)&b->d_stages, b->stages.size() * sizeof(BStage)), "cudaMalloc(batch)");
  if (!rc) rc = check_cuda(cudaMalloc((void **)&b->d_groups, std::max<size_t>(1, b->groups.size()) * sizeof(BGroup)), "cudaMalloc(batch)");
  if (!rc) rc = check_cuda(cudaMalloc((void **)&b->d_gates, std::max<size_t>(1, b->gate_tc.size()) * sizeof(BGate)), "cudaMalloc(batch)");
  if (!rc) rc = check_cuda(cudaMallocHost((void **)&b->h_gates, std::max<size_t>(1, b->gate_tc.size()) * sizeof(BGate)), "cudaMallocHost(batch)");
  if (rc) return rc;
  batch_fill_gates(b);
  // grid: CTAs per SM from the tune, but never more than fit the GPU at once;
  // a global slot for each
  int fit = 0;
  rc = batch_fit(b->tune.threads, b->tune.tile_q, &fit);
  if (rc) return rc;
  if (fit < 1) return set_error(QCS_CUDA_EUNSUP, "batch kernel does not fit an SM");
  const int grid = b->dev.num_sms * std::min(b->tune.ctas_per_sm, fit);
  // CTAs that start on an instance: 2^(n - split_q) above split_q qubits (never
  // below the tile, at most half the grid).  With CTAs joining at the end the
  // choice matters little: 384 instances of 10-22 qubits 62.8 / 62.7 / 69.8 ms
  // at split_q 27 / 19 / 16 (CTAs that wait at the stages' ends), 24 of 12-22
  // 8.8 / 8.8 / 8.6.
  for (int i = 0; i < b->count; i++) {
    BInst &I = b->insts[i];
    int G = 1;
    if (I.n > b->tune.tile_q && I.n > b->tune.split_q) {
      const int e = I.n - b->tune.split_q;
      G = e >= 20 ? (1 << 20) : (1 << e);
      G = std::min(G, std::max(1, grid / 2));
    }
    I.group = G;
    // A ticket costs two barriers and two atomics, and CTAs wait at the end of a
    // stage that leaves some of them without one: 384 instances of 10-22 qubits
    // 62.8 / 62.8 / 63.9 ms with 64 / 128 / 256 tickets, 24 of 12-22 10.5 / 8.8
    // / 8.6, 8 of 18-22 6.2 / 4.8 / 4.1, two of 21-22 3.0 / 1.8 / 1.5.
    I.tickets = b->count < grid ? 256 : 128;
  }
  // instance order
  b->order.resize(b->count);
  std::iota(b->order.begin(), b->order.end(), 0);
  if (b->tune.order == 0) {
    std::stable_sort(b->order.begin(), b->order.end(), [&](int x, int y) {
      const double cx = (double)(b->op_off[x + 1] - b->op_off[x]) * std::ldexp(1.0, b->nq[x]);
      const double cy = (double)(b->op_off[y + 1] - b->op_off[y]) * std::ldexp(1.0, b->nq[y]);
      return cx > cy;
    });
  }
  rc = check_cuda(cudaMemcpy(b->d_insts, b->insts.data(), b->insts.size() * sizeof(BInst), cudaMemcpyHostToDevice), "upload");
  if (!rc) rc = check_cuda(cudaMemcpy(b->d_stages, b->stages.data(), b->stages.size() * sizeof(BStage), cudaMemcpyHostToDevice), "upload");
  if (!rc && !b->groups.empty()) rc = check_cuda(cudaMemcpy(b->d_groups, b->groups.data(), b->groups.size() * sizeof(BGroup), cudaMemcpyHostToDevice), "upload");
  b->items.clear();
  for (int inst : b->order)
    for (int g = 0; g < b->insts[inst].group; g++) b->items.push_back(make_int2(inst, g));
  b->n_items = (int)b->items.size();
  for (int inst : b->order)
    if (b->insts[inst].n > b->tune.tile_q) b->items.push_back(make_int2(inst, 0));
  if (!rc) rc = check_cuda(cudaMalloc((void **)&b->d_items, b->items.size() * sizeof(int2)), "cudaMalloc(batch)");
  if (!rc) rc = check_cuda(cudaMemcpy(b->d_items, b->items.data(), b->items.size() * sizeof(int2), cudaMemcpyHostToDevice), "upload");
  if (rc) return rc;
  if (grid != b->grid) {
    cudaFree(b->d_slots);
    b->d_slots = nullptr;
    b->grid = grid;
    const size_t slot = b->max_n > 12 ? ((size_t)1 << b->max_n) : 4096;
    b->slot_amps = slot;
    rc = check_cuda(cudaMalloc((void **)&b->d_slots, slot * grid * sizeof(float2)), "cudaMalloc(batch slots)");
    cudaFree(b->d_sums);
    b->d_sums = nullptr;
    if (!rc) rc = check_cuda(cudaMalloc((void **)&b->d_sums, sums_of_slot(b) * grid * sizeof(double)), "cudaMalloc(batch sums)");
    if (rc) {
      b->grid = 0;  // the next schedule allocates again
      return rc;
    }
  }
  return rc;
}

static int batch_enqueue(qcs_cuda_batch *b) {
  const size_t gbytes = std::max<size_t>(1, b->gate_tc.size()) * sizeof(BGate);
  int rc = check_cuda(cudaMemcpyAsync(b->d_gates, b->h_gates, gbytes, cudaMemcpyHostToDevice, b->stream),
                      "batch gate upload");
  if (!rc) rc = check_cuda(cudaMemsetAsync(b->d_counters, 0, b->counter_bytes, b->stream), "batch counters");
  if (!rc) rc = check_cuda(cudaMemsetAsync(b->d_err, 0, sizeof(int), b->stream), "batch error flag");
  if (rc) return rc;
  const size_t smem = smem_for(b->tune.tile_q);
  const int tq = b->tune.tile_q;
  BShare *share = (BShare *)b->d_counters;
  int *queue = (int *)(share + b->count), *busy = queue + 1;
#define QCS_LAUNCH_BATCH(T)                                                                       \
  k_batch<T><<<b->grid, T, smem, b->stream>>>(                                                    \
      b->d_insts, b->d_stages, b->d_groups, b->d_gates, b->d_items, b->n_items,                     \
      (int)b->items.size() - b->n_items,                                                           \
      b->shots, b->seed, tq, b->d_slots, (i64)b->slot_amps, b->d_sums,           \
      (i64)sums_of_slot(b), queue, share, busy,                                                    \
      b->d_err, b->d_z, b->d_samples, b->wait_captured)
  switch (b->tune.threads) {
    case 256: QCS_LAUNCH_BATCH(256); break;
    case 512: QCS_LAUNCH_BATCH(512); break;
    default: QCS_LAUNCH_BATCH(1024); break;
  }
#undef QCS_LAUNCH_BATCH
  rc = check_launch("batch kernel");
  if (!rc) rc = check_cuda(cudaMemcpyAsync(b->h_z, b->d_z, b->count * sizeof(double), cudaMemcpyDeviceToHost, b->stream), "batch results");
  if (!rc && b->shots > 0)
    rc = check_cuda(cudaMemcpyAsync(b->h_samples, b->d_samples, (size_t)b->count * b->shots * sizeof(i64), cudaMemcpyDeviceToHost, b->stream), "batch samples");
  return rc;
}

static int batch_capture(qcs_cuda_batch *b) {
  b->wait_captured = wait_cycles();  // the graph's kernel node keeps this limit
  if (b->graph) {
    cudaGraphExecDestroy(b->graph);
    b->graph = nullptr;
  }
  cudaGraph_t g = nullptr;
  int rc = check_cuda(cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal), "graph capture");
  if (rc) return rc;
  int rc2 = batch_enqueue(b);
  rc = check_cuda(cudaStreamEndCapture(b->stream, &g), "graph capture end");
  if (rc2) {
    if (g) cudaGraphDestroy(g);
    return rc2;
  }
  if (rc) return rc;
  rc = check_cuda(cudaGraphInstantiate(&b->graph, g, 0), "graph instantiate");
  cudaGraphDestroy(g);
  return rc;
}

static int batch_apply_tune(qcs_cuda_batch *b, const BatchTune &t) {
  b->tune = t;
  int rc = QCS_CUDA_OK;
  if (b->planned_tile_q != t.tile_q || b->planned_regs != reg_q(t.threads))
    rc = batch_plan(b, t.tile_q, reg_q(t.threads));
  if (!rc) rc = batch_upload(b);
  if (!rc) rc = batch_capture(b);
  return rc;
}

static int batch_launch_timed(qcs_cuda_batch *b, float *ms) {
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  cudaEventRecord(e0, b->stream);
  int rc = check_cuda(cudaGraphLaunch(b->graph, b->stream), "graph launch");
  cudaEventRecord(e1, b->stream);
  if (!rc) rc = check_cuda(cudaEventSynchronize(e1), "batch sync");
  float t = 0.f;
  cudaEventElapsedTime(&t, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (ms) *ms = t;
  return rc;
}

// A timed replay whose device error flag is checked afterwards.
static int batch_launch_checked(qcs_cuda_batch *b, float *ms) {
  int rc = batch_launch_timed(b, ms);
  if (rc) return rc;
  int flag = 0;
  rc = check_cuda(cudaMemcpy(&flag, b->d_err, sizeof(int), cudaMemcpyDeviceToHost), "batch error flag");
  if (rc) return rc;
  if (flag)
    return set_error(QCS_CUDA_ETIMEOUT, "batch: a group of CTAs gave up waiting (site %d)", flag);
  return QCS_CUDA_OK;
}

static void batch_destroy(qcs_cuda_batch *b) {
  if (!b) return;
  if (b->stream) cudaStreamSynchronize(b->stream);
  batch_free_device(b);
  cudaFree(b->d_counters);
  cudaFree(b->d_z);
  cudaFree(b->d_samples);
  cudaFree(b->d_sums);
  cudaFree(b->d_slots);
  cudaFree(b->d_err);
  if (b->h_z) cudaFreeHost(b->h_z);
  if (b->h_samples) cudaFreeHost(b->h_samples);
  if (b->stream) cudaStreamDestroy(b->stream);
  delete b;
}

}  // namespace qcs

using namespace qcs;

extern "C" {

int qcs_cuda_batch_create(int count, const int *num_qubits, const int *op_offsets,
                          const qcs_cuda_op *ops, int shots, unsigned long long seed,
                          qcs_cuda_batch **out) {
  if (!out) return set_error(QCS_CUDA_EINVAL, "null out");
  *out = nullptr;
  if (count < 1 || !num_qubits || !op_offsets || (op_offsets[count] > 0 && !ops) || shots < 0)
    return set_error(QCS_CUDA_EINVAL, "bad batch arguments");
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
    cudaGetLastError();
    return set_error(QCS_CUDA_ENODEV, "no CUDA device visible");
  }
  qcs_cuda_batch *b = new qcs_cuda_batch();
  b->count = count;
  b->shots = shots;
  b->seed = seed;
  b->max_n = 0;
  b->nq.assign(num_qubits, num_qubits + count);
  b->op_off.assign(op_offsets, op_offsets + count + 1);
  b->ops.assign(ops, ops + op_offsets[count]);
  for (int i = 0; i < count; i++) {
    const int n = b->nq[i];
    if (n < 1 || n > 26 || b->op_off[i + 1] < b->op_off[i]) {
      delete b;
      return set_error(QCS_CUDA_EINVAL, "instance %d: %d qubits (1..26) or bad op range", i, n);
    }
    b->max_n = std::max(b->max_n, n);
    for (int j = b->op_off[i]; j < b->op_off[i + 1]; j++) {
      const qcs_cuda_op &o = b->ops[j];
      const bool ctl = gate_is_controlled(o.kind);
      if (!gate_kind_valid(o.kind) || o.target < 0 || o.target >= n ||
          (ctl && (o.control < 0 || o.control >= n || o.control == o.target))) {
        delete b;
        return set_error(QCS_CUDA_EINVAL, "instance %d op %d: not a valid gate", i, j);
      }
    }
  }
  int dev = 0;
  int rc = check_cuda(cudaGetDevice(&dev), "cudaGetDevice");
  if (!rc) rc = device_info(dev, &b->dev);
  if (!rc) rc = check_cuda(cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking), "cudaStreamCreate");
  // as many slots as CTAs can be resident, four to an SM at most
  b->counter_bytes = count * sizeof(BShare) + (1 + 4 * (size_t)b->dev.num_sms) * sizeof(int);
  if (!rc) rc = check_cuda(cudaMalloc((void **)&b->d_counters, b->counter_bytes), "cudaMalloc(batch)");
  if (!rc) rc = check_cuda(cudaMalloc((void **)&b->d_err, sizeof(int)), "cudaMalloc(batch)");
  if (!rc) rc = check_cuda(cudaMalloc((void **)&b->d_z, count * sizeof(double)), "cudaMalloc(batch)");
  if (!rc) rc = check_cuda(cudaMallocHost((void **)&b->h_z, count * sizeof(double)), "cudaMallocHost(batch)");
  if (!rc && shots > 0) {
    rc = check_cuda(cudaMalloc((void **)&b->d_samples, (size_t)count * shots * sizeof(i64)), "cudaMalloc(batch)");
    if (!rc) rc = check_cuda(cudaMallocHost((void **)&b->h_samples, (size_t)count * shots * sizeof(i64)), "cudaMallocHost(batch)");
  }
  BatchTune t;
  t.threads = 256;
  t.tile_q = 13;
  t.ctas_per_sm = 2;
  t.order = 0;
  t.split_q = 19;
  if (!rc) rc = batch_apply_tune(b, t);
  if (rc) {
    batch_destroy(b);
    return rc;
  }
  *out = b;
  return QCS_CUDA_OK;
}

int qcs_cuda_batch_destroy(qcs_cuda_batch *b) {
  if (!b) return set_error(QCS_CUDA_EINVAL, "null batch");
  batch_destroy(b);
  return QCS_CUDA_OK;
}

int qcs_cuda_batch_set_angles(qcs_cuda_batch *b, const double *angles) {
  if (!b || !angles) return set_error(QCS_CUDA_EINVAL, "null argument");
  int rc = check_cuda(cudaStreamSynchronize(b->stream), "batch sync");
  if (rc) return rc;
  for (size_t j = 0; j < b->ops.size(); j++) b->ops[j].angle = angles[j];
  batch_fill_gates(b);  // the captured graph uploads this pinned table on its next replay
  return QCS_CUDA_OK;
}

int qcs_cuda_batch_traffic(qcs_cuda_batch *b, double *hbm_bytes) {
  if (!b || !hbm_bytes) return set_error(QCS_CUDA_EINVAL, "null batch argument");
  double bytes = 8.0 * b->count * (1.0 + b->shots);
  for (const BInst &I : b->insts)
    if (I.n > b->planned_tile_q)  // 2 nstages - 1 stage passes, 1 read-out pass
      bytes += ldexp(8.0, I.n) * (2.0 * I.nstages);
  *hbm_bytes = bytes;
  return QCS_CUDA_OK;
}

int qcs_cuda_batch_run(qcs_cuda_batch *b, double *expect_z0, long long *samples, double *ms) {
  if (!b) return set_error(QCS_CUDA_EINVAL, "null batch");
  float t = 0.f;
  int rc = QCS_CUDA_OK;
  if (b->wait_captured != wait_cycles()) rc = batch_capture(b);  // the wait limit changed
  if (!rc) rc = batch_launch_checked(b, &t);
  if (rc) return rc;
  b->last_ms = t;
  if (ms) *ms = t;
  if (expect_z0) memcpy(expect_z0, b->h_z, b->count * sizeof(double));
  if (samples && b->shots > 0)
    memcpy(samples, b->h_samples, (size_t)b->count * b->shots * sizeof(i64));
  return QCS_CUDA_OK;
}

int qcs_cuda_batch_autotune(qcs_cuda_batch *b, int repeats, int *chosen) {
  if (!b) return set_error(QCS_CUDA_EINVAL, "null batch");
  if (repeats < 1) repeats = 1;
  auto time_tune = [&](const BatchTune &t, float *out) {
    int rc = batch_apply_tune(b, t);
    float ms = 0.f, sum = 0.f;
    if (!rc) rc = batch_launch_checked(b, &ms);  // warm-up
    for (int r = 0; !rc && r < repeats; r++) {
      rc = batch_launch_checked(b, &ms);
      sum += ms;
    }
    *out = sum / repeats;
    return rc;
  };
  const int threads[] = {256, 512, 1024};
  const int tiles[] = {12, 13, 14};
  const int ctas[] = {1, 2, 4};
  BatchTune best = b->tune;
  float best_ms = 1e30f;
  for (int th : threads)
    for (int tq : tiles) {
      int fit = 0;
      int rc = batch_fit(th, tq, &fit);
      if (rc) return rc;
      for (int cp : ctas)
        for (int ord = 0; ord < 2; ord++) {
          if (cp > fit) continue;  // it would run as a schedule of fewer
          BatchTune t = b->tune;
          t.threads = th;
          t.tile_q = tq;
          t.ctas_per_sm = cp;
          t.order = ord;
          float ms = 0.f;
          rc = time_tune(t, &ms);
          if (rc) return rc;
          if (ms < best_ms) {
            best_ms = ms;
            best = t;
          }
        }
    }
  // then how far large instances spread over CTAs (27: never)
  const int splits[] = {17, 18, 19, 20, 27};
  const BatchTune base = best;
  for (int sq : splits) {
    if (sq == base.split_q) continue;
    BatchTune t = base;
    t.split_q = sq;
    float ms = 0.f;
    int rc = time_tune(t, &ms);
    if (rc) return rc;
    if (ms < best_ms) {
      best_ms = ms;
      best = t;
    }
  }
  int rc = batch_apply_tune(b, best);
  if (rc) return rc;
  if (chosen) {
    chosen[0] = best.threads;
    chosen[1] = best.tile_q;
    chosen[2] = best.ctas_per_sm;
    chosen[3] = best.order;
  }
  return QCS_CUDA_OK;
}

int qcs_cuda_batch_split(qcs_cuda_batch *b, int split_q) {
  if (!b) return set_error(QCS_CUDA_EINVAL, "null batch");
  if (split_q < 1 || split_q > 27) return set_error(QCS_CUDA_EINVAL, "split_q %d outside 1..27", split_q);
  BatchTune t = b->tune;
  t.split_q = split_q;
  return batch_apply_tune(b, t);
}

int qcs_cuda_batch_schedule(qcs_cuda_batch *b, int *schedule) {
  if (!b || !schedule) return set_error(QCS_CUDA_EINVAL, "null argument");
  schedule[0] = b->tune.threads;
  schedule[1] = b->tune.tile_q;
  schedule[2] = std::min(b->tune.ctas_per_sm, b->grid / std::max(1, b->dev.num_sms));
  schedule[3] = b->tune.order;
  schedule[4] = b->tune.split_q;
  return QCS_CUDA_OK;
}

int qcs_cuda_batch_config(qcs_cuda_batch *b, int threads, int tile_q, int ctas_per_sm,
                          int order) {
  if (!b) return set_error(QCS_CUDA_EINVAL, "null batch");
  if ((threads != 256 && threads != 512 && threads != 1024) || tile_q < 10 || tile_q > 14 ||
      ctas_per_sm < 1 || ctas_per_sm > 4 || ctas_per_sm == 3 || order < 0 || order > 1 ||
      threads * ctas_per_sm > 1024)
    return set_error(QCS_CUDA_EINVAL, "bad batch schedule");
  if (smem_for(tile_q) * ctas_per_sm > 220 * 1024)
    return set_error(QCS_CUDA_EINVAL, "%d CTAs of tile 2^%d do not fit one SM", ctas_per_sm,
                     tile_q);
  BatchTune t = b->tune;
  t.threads = threads;
  t.tile_q = tile_q;
  t.ctas_per_sm = ctas_per_sm;
  t.order = order;
  return batch_apply_tune(b, t);
}

}  // extern "C"

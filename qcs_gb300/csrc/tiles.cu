// tiles.cu -- runs of gates applied tile by tile in shared memory.
//
// The sweeps of gates.cu read and write the whole state once per gate.  A
// plain gate list (no fusion asked for) runs here in passes instead: a pass
// takes the longest stretch of consecutive gates whose non-diagonal targets
// fit one set of tile qubits, and for every tile (one setting of the other
// qubits) a CTA reads the 2^nt amplitudes into shared memory, applies the
// stretch there and writes them back.  A diagonal gate, and the control of a
// controlled one, needs no tile qubit: outside the tile its bit is a constant
// of the tile.
//
// The gates keep their order and each amplitude goes through the same
// products and sums as in the sweeps, so the results are the sweeps' bit for
// bit; only products with an entry that is exactly 0 or 1 are left out, which
// changes no finite value (at most the sign of a zero).  A tile that holds an
// infinity or a NaN, or comes to hold one, begins again and takes every product
// the sweeps take (general_tile).
//
// Inside a tile the gates run in register groups: the stretch is cut, again
// in order, into groups whose targets lie on at most 4 tile bits; a thread
// holds the 16 amplitudes of one setting of the other bits in registers and
// takes them through the group's gates, so shared memory is read and written
// once per group.
//
// X and CNOT move amplitudes without arithmetic, and they are not even moved
// here: the shared-memory position of tile index l is an affine map over
// GF(2), A l + c, such a gate changes A or c (on the host; a CNOT whose
// control lies outside the tile changes c for half of the tiles), and the
// groups and the final store read through the map.
//
// Measured against one sweep per gate: 27 qubits complex64, brick, 752 gates
// 241 -> 22.5 ms; 13 qubits, QFT and 200 random gates 212 -> 28 us a run;
// complex128, 20 qubits, the same circuit 3.98 -> 1.78 ms.  What bounds it:
// on large complex64 states the instructions of the gate loop (a pass of 36
// rotations issues 0.69 of the slots, two fifths of them packed arithmetic,
// with DRAM at 0.39; a pass of CNOTs alone runs at 0.9 of HBM); on complex128
// the FP64 pipe (84 % busy); on small states the latency of a pass.
#include <stddef.h>
#include <string.h>

#include <algorithm>
#include <vector>

#include "common.cuh"
#include "fusion.h"
#include "tile_regs.cuh"
#include "tiles.h"

namespace qcs {

int apply_op(qcs_cuda_state *s, const qcs_cuda_op &o);

constexpr int kTileRegBits = 4;     // 16 amplitudes a thread at most
constexpr int kTileMaxBits = 11;    // tile amplitudes: 2^11 at most
constexpr int kTileMaxThreadBits = 8;
constexpr int kTileMaxGates = 128;  // per pass (they ride in the kernel parameters)
constexpr int kTileMaxGroups = 32;
constexpr int kTileMaxFlips = 32;

// How the register code applies a gate: TileGate::op.  Forms with a register
// target t come as four numbers, the phase as one for each set of register
// bits that must be set (at most two of the four).
enum TileOp {
  TO_DIAG = 0,       // + t: p0 + i p1 on bit 0, p2 + i p3 on bit 1
  TO_REAL = 4,       // + t: [[p0, p1], [p2, p3]], all real (RY; complex64: H)
  TO_PHASE = 8,      // + index of r_cond: p2 + i p3 where every condition bit is set
  TO_DIAG_OUT = 19,  // TO_DIAG with the target bit outside the registers
  TO_RX = 20,        // + t: [[p0, i p1], [i p1, p0]]
  TO_Y = 24,         // + t
  TO_HAD = 28,       // + t: p0 * [[1, 1], [1, -1]] (complex128)
  TO_SIGN = 32,      // -1 where every condition bit is set
  TO_COPY = 36,      // + t, the reference's CNOT: v0 := v1 where the control is set
  TO_NONE = 40,      // leaves finite amplitudes as they are: in no group
  TO_SWAP = 41       // X, CNOT: in the maps, never in a group
};

// One gate of a pass.  `general`: which products the sweep takes, 1: m00 v0,
// 2: m01 v1, 4: m10 v0, 8: m11 v1; an output without a product keeps its
// value.
template <typename R> struct TileGate {
  R p[4];
  uint32_t id_cond;       // bits of the tile's id that must be set
  uint32_t id_tgt;        // the target, where it is a bit of the tile's id
  unsigned short t_cond;  // bits of the thread index that must be set
  unsigned short t_tgt;   // the target, where it is a bit of the thread index
  unsigned short l_tgt, l_ctl;  // target and control as tile bits
  uint32_t id_ctl;              // control as a bit of the tile's id
  unsigned char r_cond;   // register bits that must be set
  unsigned char op;       // TileOp
  unsigned char general;
  unsigned char pad;
};

// A group: gates [gate0, gate1) on registers e, where bit j of e adds
// reg[j], bit j of the thread index col[j], to the shared-memory position
// (XOR).  Before it, flips [flip0, flip1) change the constant.
// (reg: 32 bits wide because with 16 one build of k_tile took reg[3] for 0.)
struct TileGroup {
  unsigned char gate0, gate1, flip0, flip1;
  int reg[kTileRegBits];
  unsigned short col[kTileMaxThreadBits];
};
struct TileFlip {
  unsigned short mask;  // XORed into the constant
  short id_bit;         // where this bit of the tile's id is set (-1: always)
};

template <typename R> struct TilePass {
  i64 n_tiles;
  R minus_zero;  // see tile_regs.cuh
  int nt, nout, ngroups, ngates;
  unsigned char flip0, flip1;       // flips before the store
  signed char q[kTileMaxBits];      // tile bit -> qubit, ascending
  signed char out[36];              // bit of the tile id -> qubit, ascending
  unsigned short store[kTileMaxBits];  // tile bit -> position, after the last gate
  TileFlip flip[kTileMaxFlips];
  TileGroup group[kTileMaxGroups];
  // the gates of the groups, one group after another, then the others;
  // order: all of them as the list has them
  unsigned char order[kTileMaxGates];
  TileGate<R> gate[kTileMaxGates];
};

// ---------------------------------------------------------------------------
// device
// ---------------------------------------------------------------------------

// Collects whether an amplitude was an infinity or a NaN: 0 * x is NaN for
// those alone (and FP32 products cost no integer slot); FP64, whose products
// are dear, looks at the exponent.
struct FiniteF32 {
  float z = 0.f;
  __device__ __forceinline__ void see(float2 a) { z = fmaf(a.x, 0.f, fmaf(a.y, 0.f, z)); }
  __device__ __forceinline__ bool bad() const { return z != 0.f; }
};
struct FiniteF64 {
  bool b = false;
  __device__ __forceinline__ void see(double2 a) {
    b = b || (__double2hiint(a.x) & 0x7ff00000) == 0x7ff00000 ||
        (__double2hiint(a.y) & 0x7ff00000) == 0x7ff00000;
  }
  __device__ __forceinline__ bool bad() const { return b; }
};

// max_bits: a tile's qubits.  Measured, 11 against 12 (complex64): 27.0 and 29.2
// ms on 27 qubits (brick, 752 gates), 87 and 101 us on 13, where the threads
// of the tiles are all the parallelism there is; 10 against 11 (complex128,
// 20 qubits, 417 gates): 2.13 and 2.32 ms.  Likewise 16 amplitudes a thread
// against 32: 27.7 and 28.9 ms, 87 and 122 us.  (By number of tiles: run_tiles.)
// low: qubits every tile holds, so that it is read in runs of 128 bytes.
// blocks: CTAs an SM holds at 16 amplitudes a thread.  complex64: 72 registers, for
// which 140 bytes a thread are spilled outside the loop over gates (2.6 M of a 26-qubit
// pass's 290 M warp instructions); the bound was chosen when the grid was what the GPU
// holds at once.
template <typename C> struct TileTraits;
template <> struct TileTraits<float2> {
  typedef float R;
  typedef float Elem;  // of the tile in shared memory
  typedef FiniteF32 Finite;
  template <int RB> using Regs = RegsF32<RB>;
  static constexpr int max_bits = 11, low = 4, blocks = 7;
};
template <> struct TileTraits<double2> {
  typedef double R;
  typedef double2 Elem;
  typedef FiniteF64 Finite;
  template <int RB> using Regs = RegsF64<RB>;
  static constexpr int max_bits = 10, low = 3, blocks = 8;
};

#define QCS_TILE_TARGET(CALL)                                               \
  if (Regs::N > 4 && (op & 2)) {                                            \
    if (Regs::N > 8 && (op & 1)) { constexpr int TB = Regs::N > 8 ? 3 : 0; CALL; } \
    else { constexpr int TB = Regs::N > 4 ? 2 : 0; CALL; }                  \
  } else {                                                                  \
    if (op & 1) { constexpr int TB = 1; CALL; }                             \
    else { constexpr int TB = 0; CALL; }                                    \
  }
#define QCS_TILE_PHASE(I, COND)                   \
  case TO_PHASE + I:                              \
    if constexpr (COND < Regs::N) a.template phase<COND>(g.p); \
    break;

// One gate on the amplitudes of thread t.  (The compiler makes no jump table of
// a switch here but a tree of comparisons over all the forms, seven branches
// a gate; asking for the common classes first takes four.)
template <typename Regs, typename R>
__device__ __forceinline__ void tile_apply(Regs &a, const TileGate<R> &g, uint32_t t,
                                           uint32_t tile, u64 z) {
  const int op = g.op;
  if (op < TO_REAL) {
    QCS_TILE_TARGET((a.template diag<TB>(g.p)))
  } else if (op < TO_PHASE) {
    QCS_TILE_TARGET((a.template real<TB>(g.p, z)))
  } else if (op == TO_DIAG_OUT) {
    const bool one = (t & g.t_tgt) || (tile & g.id_tgt);
    const R f[2] = {one ? g.p[2] : g.p[0], one ? g.p[3] : g.p[1]};
    a.template phase<0>(f);
  } else if ((t & g.t_cond) != g.t_cond || (tile & g.id_cond) != g.id_cond) {
    // a form with a condition that is not met (the others have none)
  } else if (op < TO_DIAG_OUT) {
    switch (op) {
      QCS_TILE_PHASE(0, 0) QCS_TILE_PHASE(1, 1) QCS_TILE_PHASE(2, 2) QCS_TILE_PHASE(3, 3)
      QCS_TILE_PHASE(4, 4) QCS_TILE_PHASE(5, 5) QCS_TILE_PHASE(6, 6) QCS_TILE_PHASE(7, 8)
      QCS_TILE_PHASE(8, 9) QCS_TILE_PHASE(9, 10) QCS_TILE_PHASE(10, 12)
    }
  } else if (op < TO_Y) {
    QCS_TILE_TARGET((a.template rx<TB>(g.p, z)))
  } else if (op < TO_HAD) {
    QCS_TILE_TARGET((a.template y<TB>()))
  } else if (op < TO_SIGN) {
    if constexpr (sizeof(R) == 8) QCS_TILE_TARGET((a.template had<TB>(g.p)))
  } else if (op < TO_COPY) {
    a.sign(g.r_cond);
  } else {
    QCS_TILE_TARGET((a.template copy<TB>(g.r_cond)))
  }
}
#undef QCS_TILE_PHASE
#undef QCS_TILE_TARGET

// d * v with the sweeps' rounding (tile_regs.cuh).
__device__ __forceinline__ float2 turn(float2 d, float2 v) {
  return make_float2(__fmaf_rn(d.x, v.x, -__fmul_rn(d.y, v.y)),
                     __fmaf_rn(d.y, v.x, __fmul_rn(d.x, v.y)));
}
__device__ __forceinline__ double2 turn(double2 d, double2 v) { return cmul(d, v); }

// A gate's 2x2 from its record.
template <typename C, typename R>
__device__ void tile_matrix(const TileGate<R> &g, C (&m)[4]) {
  const int op = g.op;
  if (op < TO_REAL || op == TO_DIAG_OUT) {
    m[0].x = g.p[0];
    m[0].y = g.p[1];
    m[3].x = g.p[2];
    m[3].y = g.p[3];
  } else if (op < TO_PHASE || (op >= TO_HAD && op < TO_SIGN)) {
    for (int i = 0; i < 4; i++) m[i].x = g.p[i];
  } else if (op < TO_DIAG_OUT) {
    m[0].x = 1;
    m[3].x = g.p[0];
    m[3].y = g.p[1];
  } else if (op < TO_Y) {
    m[0].x = m[3].x = g.p[0];
    m[1].y = m[2].y = g.p[1];
  } else if (op < TO_HAD) {
    m[1].y = -1;
    m[2].y = 1;
  } else if (op < TO_COPY) {
    m[0].x = 1;
    m[3].x = -1;
  } else if (op == TO_NONE) {  // the identity; the reference's CPHASE takes its 1 alone
    m[0].x = m[3].x = 1;
  } else {
    m[1].x = m[2].x = 1;
  }
}

// The gates of a pass on a tile with an infinity or a NaN in it: one at a
// time, with the products the sweep of each gate takes (TileGate::general),
// so that what spreads, and where to, is the same.
__device__ __forceinline__ float2 sum2(float2 v, float2 w) {
  return make_float2(__fadd_rn(v.x, w.x), __fadd_rn(v.y, w.y));
}
__device__ __forceinline__ double2 sum2(double2 v, double2 w) { return cadd(v, w); }

template <typename C, typename E, typename R>
__device__ __noinline__ void general_tile(E *S, const TilePass<R> &P, uint32_t tile) {
  const C kind = {};
  const int L = 1 << P.nt;
  for (int gi = 0; gi < P.ngates; gi++) {
    const TileGate<R> &g = P.gate[P.order[gi]];
    C m[4] = {};
    tile_matrix(g, m);
    if ((tile & g.id_ctl) == g.id_ctl) {
      for (int l = threadIdx.x; l < L; l += blockDim.x) {
        if ((l & g.l_ctl) != g.l_ctl) continue;
        const int x = tile_pos(l, kind);
        if (!g.l_tgt) {  // a diagonal on a qubit outside the tile
          const bool one = tile & g.id_tgt;
          if (g.general & (one ? 8 : 1))
            tile_put(S, L, x, turn(one ? m[3] : m[0], tile_get(S, L, x)));
          continue;
        }
        if (l & g.l_tgt) continue;
        const int y = tile_pos(l | g.l_tgt, kind);
        const C v0 = tile_get(S, L, x), v1 = tile_get(S, L, y);
        const int u = g.general & 3, w = g.general >> 2;
        if (u)
          tile_put(S, L, x, u == 3 ? sum2(turn(m[0], v0), turn(m[1], v1))
                                   : u == 1 ? turn(m[0], v0) : turn(m[1], v1));
        if (w)
          tile_put(S, L, y, w == 3 ? sum2(turn(m[2], v0), turn(m[3], v1))
                                   : w == 1 ? turn(m[2], v0) : turn(m[3], v1));
      }
    }
    __syncthreads();
  }
}

// One thread per 2^RB amplitudes of the tile; CTAs are persistent
// over their tiles.
template <typename C, int RB>
__global__ void __launch_bounds__(1 << (TileTraits<C>::max_bits - RB),
                                  TileTraits<C>::blocks >> (kTileRegBits - RB))
    k_tile(C *v, const __grid_constant__ TilePass<typename TileTraits<C>::R> P) {
  typedef typename TileTraits<C>::Elem E;
  constexpr int REGS = 1 << RB;
  constexpr int UNIT = 16 / sizeof(C);  // amplitudes per 16-byte access
  constexpr int STEPS = REGS / UNIT;    // accesses per thread and tile
  constexpr int STEP_BITS = UNIT == 2 ? RB - 1 : RB;
  const C kind = {};
  if constexpr (sizeof(C) == 8) QCS_REGS_F32_DECLARE(8);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  E *S = reinterpret_cast<E *>(smem_raw);
  const int L = 1 << P.nt;
  const u64 z = both2((float)P.minus_zero);
  const int t = threadIdx.x;
  const int sb = P.nt - STEP_BITS;  // the tile bits from sb up count a thread's accesses
  // this thread's first unit: its offset in memory, its position on loading
  // and (by the map left by the last gate) on storing
  i64 toff = 0;
  int tstore = 0;
  for (int m = 0; m < sb; m++)
    if ((t * UNIT >> m) & 1) {
      toff |= 1LL << P.q[m];
      tstore ^= P.store[m];
    }
  const int tload = tile_pos(t * UNIT, kind);
  auto step_off = [&](int k) {
    i64 o = 0;
#pragma unroll
    for (int j = 0; j < STEP_BITS; j++)
      if ((k >> j) & 1) o |= 1LL << P.q[sb + j];
    return o;
  };
  auto step_store = [&](int k) {
    int o = 0;
#pragma unroll
    for (int j = 0; j < STEP_BITS; j++)
      if ((k >> j) & 1) o ^= P.store[sb + j];
    return o;
  };
  grid_wait();
  for (i64 tile = blockIdx.x; tile < P.n_tiles; tile += gridDim.x) {
    i64 base = 0;
    for (int j = 0; j < P.nout; j++) base |= ((tile >> j) & 1LL) << P.out[j];
    C *const vt = v + base + toff;
    const uint32_t id = (uint32_t)tile;
    // Of an infinity, in the tile from the start or come up on the way, the
    // products with zeros that are left out here are NaNs in the sweeps.  Some
    // amplitude is an infinity or a NaN to the end then (nothing but the
    // reference's CNOT drops one, and that drops the same ones in the sweeps), so
    // one look after the last gate finds it, while the tile is still in memory to
    // begin again.  The look is taken where it costs least: large states, bound by
    // instructions, in the registers of the last group (27 qubits 24.1 -> 22.5 ms
    // against a look at every amplitude that is read, in the units of the store
    // 24.8), small ones, bound by latency, in the units of the store (16 qubits
    // 189 -> 186 us a run with its read-outs, in the registers 191).
    bool bad = false;
    {
      uint4 x[STEPS];
#pragma unroll
      for (int k = 0; k < STEPS; k++) x[k] = *reinterpret_cast<const uint4 *>(vt + step_off(k));
#pragma unroll
      for (int k = 0; k < STEPS; k++) {
        const C *y = reinterpret_cast<const C *>(&x[k]);
        const int at = tload ^ tile_pos(k << sb, kind);
#pragma unroll
        for (int j = 0; j < UNIT; j++) tile_put(S, L, at ^ j, y[j]);
      }
    }
    __syncthreads();
    int c = 0;  // the map's constant
    auto flips = [&](int f0, int f1) {
      for (int f = f0; f < f1; f++)
        if (P.flip[f].id_bit < 0 || ((id >> P.flip[f].id_bit) & 1)) c ^= P.flip[f].mask;
    };
    for (int gr = 0; gr < P.ngroups; gr++) {
      const TileGroup &G = P.group[gr];
      flips(G.flip0, G.flip1);
      int at = c;
#pragma unroll
      for (int j = 0; j < TileTraits<C>::max_bits - RB; j++)
        if ((t >> j) & 1) at ^= G.col[j];
      auto place = [&](int (&pos)[REGS]) {  // register e: its bits' columns
        int lo[4], hi[REGS / 4];
#pragma unroll
        for (int k = 0; k < 4; k++)
          lo[k] = at ^ ((k & 1) ? G.reg[0] : 0) ^ ((k & 2) ? G.reg[1] : 0);
#pragma unroll
        for (int k = 0; k < REGS / 4; k++)
          hi[k] = ((k & 1) ? G.reg[2] : 0) ^ ((k & 2) ? G.reg[3] : 0);
#pragma unroll
        for (int e = 0; e < REGS; e++) pos[e] = lo[e & 3] ^ hi[e >> 2];
      };
      typename TileTraits<C>::template Regs<RB> a;
      {
        int pos[REGS];
        place(pos);
        a.load(S, L, pos);
      }
      for (int i = G.gate0; i < G.gate1; i++) tile_apply(a, P.gate[i], (uint32_t)t, id, z);
      asm volatile("" : "+r"(at));  // the positions are formed anew, not kept
      int pos[REGS];
      place(pos);
      if constexpr (RB == kTileRegBits) {
        if (gr + 1 == P.ngroups) {
          bad = __syncthreads_or(a.store_finite(S, L, pos));
          break;
        }
      }
      a.store(S, L, pos);
      __syncthreads();
    }
    flips(P.flip0, P.flip1);
    if constexpr (RB < kTileRegBits) {
      uint4 x[STEPS];
      typename TileTraits<C>::Finite fin;
#pragma unroll
      for (int k = 0; k < STEPS; k++) {
        C *y = reinterpret_cast<C *>(&x[k]);
        const int at = c ^ tstore ^ step_store(k);
#pragma unroll
        for (int j = 0; j < UNIT; j++) {
          y[j] = tile_get(S, L, j ? at ^ P.store[0] : at);
          fin.see(y[j]);
        }
      }
      bad = __syncthreads_or(fin.bad());
      if (!bad) {
#pragma unroll
        for (int k = 0; k < STEPS; k++) *reinterpret_cast<uint4 *>(vt + step_off(k)) = x[k];
        continue;  // no access to shared memory since the barrier
      }
    } else if (!bad) {
#pragma unroll
      for (int k = 0; k < STEPS; k++) {
        uint4 x;
        C *y = reinterpret_cast<C *>(&x);
        const int at = c ^ tstore ^ step_store(k);
#pragma unroll
        for (int j = 0; j < UNIT; j++) y[j] = tile_get(S, L, j ? at ^ P.store[0] : at);
        *reinterpret_cast<uint4 *>(vt + step_off(k)) = x;
      }
    }
    if (bad) {
      for (int k = 0; k < STEPS; k++) {
        const uint4 x = *reinterpret_cast<const uint4 *>(vt + step_off(k));
        const C *y = reinterpret_cast<const C *>(&x);
        for (int j = 0; j < UNIT; j++) tile_put(S, L, tload ^ tile_pos((k << sb) | j, kind), y[j]);
      }
      __syncthreads();
      general_tile<C>(S, P, id);
      for (int k = 0; k < STEPS; k++) {
        uint4 x;
        C *y = reinterpret_cast<C *>(&x);
        for (int j = 0; j < UNIT; j++)
          y[j] = tile_get(S, L, tload ^ tile_pos((k << sb) | j, kind));
        *reinterpret_cast<uint4 *>(vt + step_off(k)) = x;
      }
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// host: the plan
// ---------------------------------------------------------------------------

// The qubit a gate needs in the tile: the target of a non-diagonal gate; -1
// for a diagonal one.
static int needed_qubit(const qcs_cuda_op &o) {
  switch (o.kind) {
    case QCS_GATE_H: case QCS_GATE_X: case QCS_GATE_Y: case QCS_GATE_RX: case QCS_GATE_RY:
    case QCS_GATE_CNOT: return o.target;
    default: return -1;
  }
}

static bool moves_only(const qcs_cuda_op &o, bool reference) {
  return o.kind == QCS_GATE_X || (o.kind == QCS_GATE_CNOT && !reference);
}

// The register groups of a stretch.  A move (X, CNOT) waits for the end of
// the current group; a later gate may still join the group if it commutes
// with the waiting moves exactly: on other qubits, or diagonal on their
// controls.  Stops early (s.last) when the pass is full.
static void cut_groups(const qcs_cuda_op *ops, bool reference, int regs, TileStretch &s) {
  typedef unsigned long long Mask;
  Mask moved = 0, ctl = 0;  // targets and controls of the waiting moves
  TileStretch::Group g;
  int flips = 0;
  auto close = [&](int at) {
    if (g.gates.empty() && g.moves.empty()) return true;
    if ((int)s.groups.size() == kTileMaxGroups - 1 || flips > kTileMaxFlips - 2) {
      s.last = at;
      return false;
    }
    s.groups.push_back(g);
    g = TileStretch::Group();
    moved = ctl = 0;
    return true;
  };
  for (int i = s.first; i < s.last; i++) {
    const qcs_cuda_op &o = ops[i];
    const Mask t = 1ULL << o.target;
    const Mask c = gate_is_controlled(o.kind) ? 1ULL << o.control : 0;
    if (moves_only(o, reference)) {
      if (flips > kTileMaxFlips - 2) {
        s.last = i;
        break;
      }
      if (!c || !(s.qubits & c)) flips++;  // at most one flip each
      g.moves.push_back(i);
      moved |= t;
      ctl |= c;
      continue;
    }
    const int q = needed_qubit(o);
    const bool held = q < 0 || ((g.qubits >> q) & 1);
    const bool full = !held && __builtin_popcountll(g.qubits) == regs;
    // a condition of the gate on a moved qubit, or its target on a control
    const bool clash = ((t | c) & moved) || (q >= 0 && (t & ctl));
    if ((full || clash) && !close(i)) break;
    if (q >= 0) g.qubits |= 1ULL << q;
    g.gates.push_back(i);
  }
  s.groups.push_back(g);
}

std::vector<TileStretch> tile_stretches(const qcs_cuda_op *ops, int count, int n, int nt, int low,
                                        bool reference, int regs) {
  std::vector<TileStretch> plan;
  for (int i = 0; i < count;) {
    TileStretch s;
    s.first = i;
    unsigned long long set = (1ULL << low) - 1;
    int room = nt - low;
    for (; i < count && i - s.first < kTileMaxGates; i++) {
      const int q = needed_qubit(ops[i]);
      if (q < 0 || ((set >> q) & 1)) continue;
      if (room == 0) break;
      set |= 1ULL << q;
      room--;
    }
    for (int q = low; q < n && room > 0; q++)
      if (!((set >> q) & 1)) {
        set |= 1ULL << q;
        room--;
      }
    s.last = i;
    s.qubits = set;
    cut_groups(ops, reference, regs, s);
    i = s.last;
    plan.push_back(s);
  }
  return plan;
}

// Which products the sweep of this gate takes (gates.cu), as TileGate::general.
static int sweep_products(const qcs_cuda_state *s, const double m[8], bool controlled) {
  auto zero = [&](int i) { return m[2 * i] == 0.0 && m[2 * i + 1] == 0.0; };
  auto one = [&](int i) { return m[2 * i] == 1.0 && m[2 * i + 1] == 0.0; };
  const bool diag = zero(1) && zero(2), exch = zero(0) && zero(3);
  if (s->sem == QCS_CUDA_REFERENCE) {
    if (controlled) return zero(1) ? 1 : zero(0) ? 2 : 3;
    return diag ? 1 | 8 : exch ? 2 | 4 : 15;
  }
  if (diag && one(0)) return one(3) ? 0 : 8;
  if (!controlled && diag) return 1 | 8;
  if (exch && s->prec == QCS_CUDA_C128) return 2 | 4;
  return 15;
}

// The constants of a record from the gate's 2x2.
template <typename R>
static void fill_const(TileGate<R> &g, int op, const double m[8]) {
  if (op == TO_DIAG || op == TO_DIAG_OUT) {
    for (int i = 0; i < 2; i++) {
      g.p[i] = (R)m[i];
      g.p[2 + i] = (R)m[6 + i];
    }
  } else if (op == TO_REAL || op == TO_HAD) {
    for (int i = 0; i < 4; i++) g.p[i] = (R)m[2 * i];
  } else if (op == TO_RX) {
    g.p[0] = (R)m[0];
    g.p[1] = (R)m[3];
  } else if (op == TO_PHASE) {
    g.p[0] = (R)m[6];
    g.p[1] = (R)m[7];
  }
}

// Gate record; bit_of: qubit -> tile bit (-1: outside), id_of: qubit -> bit of
// the tile's id, reg_of and thread_of: tile bit -> register or thread bit of
// the gate's group (-1: the other).
template <typename R>
static void fill_gate(const qcs_cuda_state *s, const qcs_cuda_op &o, const int *bit_of,
                      const int *id_of, const int *reg_of, const int *thread_of, TileGate<R> &g) {
  memset(&g, 0, sizeof(g));
  double m[8];
  gate_matrix(o.kind, o.angle, m);
  const bool ctl = gate_is_controlled(o.kind);
  const bool ref = s->sem == QCS_CUDA_REFERENCE;
  g.general = (unsigned char)sweep_products(s, m, ctl);
  if (bit_of[o.target] >= 0) g.l_tgt = (unsigned short)(1 << bit_of[o.target]);
  else g.id_tgt = 1u << id_of[o.target];
  if (ctl) {
    if (bit_of[o.control] >= 0) g.l_ctl = (unsigned short)(1 << bit_of[o.control]);
    else g.id_ctl = 1u << id_of[o.control];
  }
  auto place = [&](int q, unsigned char &r, unsigned short &t, uint32_t &id) {
    if (bit_of[q] < 0) id |= 1u << id_of[q];
    else if (reg_of[bit_of[q]] >= 0) r |= (unsigned char)(1 << reg_of[bit_of[q]]);
    else t |= (unsigned short)(1 << thread_of[bit_of[q]]);
  };
  int op = TO_NONE;
  bool cond_tgt = false;  // the target bit is a condition too (phases)
  switch (o.kind) {
    case QCS_GATE_H: op = sizeof(R) == 8 ? TO_HAD : TO_REAL; break;
    case QCS_GATE_RY: op = TO_REAL; break;
    case QCS_GATE_RX: op = TO_RX; break;
    case QCS_GATE_X: op = TO_SWAP; break;
    case QCS_GATE_Y: op = TO_Y; break;
    case QCS_GATE_CNOT: op = ref ? TO_COPY : TO_SWAP; break;
    case QCS_GATE_RZ: op = TO_DIAG; break;
    case QCS_GATE_Z: op = TO_SIGN; cond_tgt = true; break;
    case QCS_GATE_P: op = TO_PHASE; cond_tgt = true; break;
    // under the reference's rule a CPHASE multiplies by its U00 = 1 only
    case QCS_GATE_CPHASE: op = ref ? TO_NONE : TO_PHASE; cond_tgt = true; break;
    default: break;  // identity
  }
  if (ctl) place(o.control, g.r_cond, g.t_cond, g.id_cond);
  if (cond_tgt) place(o.target, g.r_cond, g.t_cond, g.id_cond);
  const int reg = bit_of[o.target] >= 0 ? reg_of[bit_of[o.target]] : -1;
  if (op == TO_DIAG && reg < 0) {
    op = TO_DIAG_OUT;
    unsigned char no_reg = 0;
    uint32_t id = 0;  // id_tgt is set above
    place(o.target, no_reg, g.t_tgt, id);
  }
  fill_const(g, op, m);
  static const unsigned char conds[11] = {0, 1, 2, 3, 4, 5, 6, 8, 9, 10, 12};
  if (op == TO_PHASE) op += (int)(std::find(conds, conds + 11, g.r_cond) - conds);
  if (op == TO_DIAG || op == TO_REAL || op == TO_RX || op == TO_Y || op == TO_HAD || op == TO_COPY)
    op += reg;
  g.op = (unsigned char)op;
}

template <typename C, int RB>
static int launch_pass(qcs_cuda_state *s, const qcs_cuda_op *ops, const TileStretch &st) {
  typedef typename TileTraits<C>::R R;
  const C kind = {};
  TilePass<R> P;
  memset(&P, 0, offsetof(TilePass<R>, gate));
  int bit_of[36], id_of[36];
  for (int q = 0; q < s->n; q++) {
    bit_of[q] = id_of[q] = -1;
    if ((st.qubits >> q) & 1) {
      bit_of[q] = P.nt;
      P.q[P.nt++] = (signed char)q;
    } else {
      id_of[q] = P.nout;
      P.out[P.nout++] = (signed char)q;
    }
  }
  P.n_tiles = 1LL << P.nout;
  P.minus_zero = (R)-0.0;
  P.ngates = st.last - st.first;
  int map[kTileMaxBits];  // column b: what tile bit b adds to the position
  for (int b = 0; b < P.nt; b++) map[b] = tile_pos(1 << b, kind);
  int nrun = 0, nrest = P.ngates, nflip = 0, flip0 = 0;
  auto move = [&](const qcs_cuda_op &o) {  // X or CNOT: see the head of the file
    const int t = bit_of[o.target];
    if (o.kind == QCS_GATE_CNOT && bit_of[o.control] >= 0) {
      map[bit_of[o.control]] ^= map[t];
    } else {
      TileFlip &f = P.flip[nflip++];
      f.mask = (unsigned short)map[t];
      f.id_bit = (short)(o.kind == QCS_GATE_CNOT ? id_of[o.control] : -1);
    }
  };
  int none[kTileMaxBits];
  std::fill(none, none + kTileMaxBits, 0);
  for (const TileStretch::Group &gr : st.groups) {
    if (!gr.gates.empty()) {
      TileGroup &G = P.group[P.ngroups++];
      G.flip0 = (unsigned char)flip0;
      G.flip1 = (unsigned char)nflip;
      flip0 = nflip;
      // Which tile bits the registers take besides the group's targets, and
      // which the lanes of a warp: a condition on a register bit costs the
      // other registers nothing and one on the upper thread bits skips whole
      // warps, but one on a lane leaves half of the warp idle, so the bits
      // that most gates depend on come first.
      int uses[kTileMaxBits] = {0}, order[kTileMaxBits];
      for (int i : gr.gates) {
        const qcs_cuda_op &o = ops[i];
        if (bit_of[o.target] >= 0) uses[bit_of[o.target]]++;
        if (gate_is_controlled(o.kind) && bit_of[o.control] >= 0) uses[bit_of[o.control]]++;
      }
      for (int b = 0; b < P.nt; b++) {
        order[b] = P.nt - 1 - b;
        if ((gr.qubits >> P.q[b]) & 1) uses[b] += 1 << 16;  // a target: in a register
      }
      std::stable_sort(order, order + P.nt, [&](int x, int y) { return uses[x] > uses[y]; });
      int reg_of[kTileMaxBits], thread_of[kTileMaxBits];
      std::fill(reg_of, reg_of + kTileMaxBits, -1);
      std::fill(thread_of, thread_of + kTileMaxBits, -1);
      for (int j = 0; j < P.nt; j++) {
        const int b = order[j];
        if (j < RB) {  // the least used one is the pair bit (tile_regs.cuh)
          G.reg[RB - 1 - j] = map[b];
          reg_of[b] = RB - 1 - j;
        } else {
          const int t = P.nt - 1 - j;  // the last, least used ones are the lanes
          G.col[t] = (unsigned short)map[b];
          thread_of[b] = t;
        }
      }
      G.gate0 = (unsigned char)nrun;
      for (int i : gr.gates) {
        TileGate<R> g;
        fill_gate<R>(s, ops[i], bit_of, id_of, reg_of, thread_of, g);
        const int at = g.op != TO_NONE ? nrun++ : --nrest;
        P.gate[at] = g;
        P.order[i - st.first] = (unsigned char)at;
      }
      G.gate1 = (unsigned char)nrun;
    }
    for (int i : gr.moves) {
      const int at = --nrest;
      fill_gate<R>(s, ops[i], bit_of, id_of, none, none, P.gate[at]);
      P.order[i - st.first] = (unsigned char)at;
      move(ops[i]);
    }
  }
  if (RB == kTileRegBits && P.ngroups == 0) {  // moves alone: the look takes a group
    TileGroup &G = P.group[P.ngroups++];
    for (int j = 0; j < P.nt; j++) {
      if (j < RB) G.reg[RB - 1 - j] = map[P.nt - 1 - j];
      else G.col[P.nt - 1 - j] = (unsigned short)map[P.nt - 1 - j];
    }
  }
  P.flip0 = (unsigned char)flip0;
  P.flip1 = (unsigned char)nflip;
  for (int b = 0; b < P.nt; b++) P.store[b] = (unsigned short)map[b];
  const int threads = 1 << (P.nt - RB);
  const size_t smem = sizeof(C) << P.nt;
  // Several times the CTAs that an SM holds: CTAs that end and begin fall out of
  // step, so the loads of some run under the gates of others, and the last tiles
  // are spread.  As many as it holds (7), 28, 64, 100: 27 qubits (complex64, 752
  // gates) 27.7, 25.7, 25.1, 24.9 ms alone, but 23.9, 24.0, 24.3 a run where
  // three states run at once, which has the same effect; 24 qubits 3.13, 2.89,
  // 2.97, 2.97.  complex128, 24 qubits (8, 28, 100) 33.8, 32.4, 31.9.
  const i64 cap = (i64)s->dev.num_sms * (sizeof(C) == 8 ? 28 : 64);
  const int grid = (int)std::min<i64>(P.n_tiles, cap);
  s->h2d_bytes += (long long)(offsetof(TilePass<R>, gate) + P.ngates * sizeof(TileGate<R>));
  prof_begin(s);
  // Started early (launch_next) where every tile finds an SM of its own, and
  // for complex64 but not at one to three tiles an SM: new angles every run,
  // 16 qubits (32 tiles) 99 -> 76 us, 18 (128) 108 -> 89, 20 (512) 186 -> 153;
  // 19 (256), replayed, 105 -> 125; complex128, 18 qubits (256) 610 -> 1101.
  const int sms = s->dev.num_sms;
  const bool early = 2 * grid <= sms || (sizeof(C) == 8 && (grid <= sms || grid > 3 * sms));
  launch_next(early, k_tile<C, RB>, grid, threads, smem, s->stream, (C *)s->vec, P);
  invalidate_sum(s);
  return launched(s, KC_TILE, 2.0 * s->size * sizeof(C), "gate tile pass");
}

// Whether the sweeps of a stretch's gates cost less than its pass: a sweep leaves
// out what its gate leaves alone, the whole of an identity's, three quarters of a
// controlled phase's, half of a phase's or a CNOT's.  A pass reads and writes
// everything once.  Work is counted in sixteenths of a pass; a condition on a
// qubit so low that its amplitudes lie in the same 32 bytes as the others saves
// nothing, in the same 128 bytes part of it.  The reference's sweeps go out of
// place, over everything.
// complex64, us by sweeps against us by a pass: two controlled phases on 20, 22, 23,
// 24, 27, 30 qubits 8, 9, 12, 17, 175, 1299 against 5, 11, 21, 47, 335, 2660; four 17,
// 20, 25, 40, 350, 2597 against 5, 12, 23, 46, 340, 2650; two phases 8, 12, 17, 33,
// 335, 2596 against the same.  Below 32 MB the launches decide, above 64 the bytes
// (that lie in L2 in part: 128 MB), between them both.
// complex128: the FP64 pipe bounds both ways, and a pass has its reads and writes on
// top; but it takes signs and moves without that pipe, and is better at all else.
// Two controlled phases on 18, 20, 22, 27 qubits 12, 14, 33, 784 against 10, 17, 43,
// 1058, on the lowest qubits of 21, 23, 27 21, 72, 1129 against 24, 81, 1060; four 25,
// 29, 66, 1568 against 12, 27, 67, 1740; three phases 19, 31, 86, 2331 against 13, 26,
// 81, 2450; two CNOTs 16, 21, 57, 1556 against 5, 8, 18, 638.
static bool sweeps_cost_less(const qcs_cuda_state *s, const qcs_cuda_op *ops, int count) {
  if (s->sem == QCS_CUDA_REFERENCE) return false;
  const bool c64 = s->prec == QCS_CUDA_C64;
  const i64 bytes = s->size * (c64 ? 8 : 16);
  const int sector = c64 ? 2 : 1;  // qubits within 32 bytes
  int sweeps = 0, work = 0;
  for (int i = 0; i < count && work <= 32; i++) {
    const qcs_cuda_op &o = ops[i];
    double m[8];
    gate_matrix(o.kind, o.angle, m);
    auto is = [&](int e, double v) { return m[2 * e] == v && m[2 * e + 1] == 0.0; };
    const bool diag = is(1, 0.0) && is(2, 0.0), ctl = gate_is_controlled(o.kind);
    if (diag && is(0, 1.0) && is(3, 1.0)) continue;  // an identity: no sweep
    if (!c64 && !diag) return false;
    if (!c64 && o.kind == QCS_GATE_Z) return false;
    int w = 16;
    auto condition = [&](int q) { w = q < sector ? w : q < sector + 2 ? w * 3 / 4 : w / 2; };
    if (ctl) condition(o.control);
    if (diag && is(0, 1.0)) condition(o.target);
    work += w;
    sweeps++;
  }
  if (sweeps <= 1) return true;
  if (c64) {
    if (bytes < (32 << 20)) return false;
    if (bytes <= (64 << 20)) return 4 * sweeps + work <= (bytes <= (32 << 20) ? 20 : 28);
    return work <= 16;
  }
  if (bytes < (16 << 20)) return false;
  if (sweeps == 2 && bytes >= (32 << 20) && bytes <= (128 << 20)) return work <= 24;
  return work <= (bytes < (64 << 20) ? 12 : bytes < (128 << 20) ? 16 : 20);
}

template <typename C, int RB>
static int run_tiles_t(qcs_cuda_state *s, const qcs_cuda_op *ops, int count, int bits) {
  const int nt = std::min(bits, s->n);
  for (const TileStretch &st : tile_stretches(ops, count, s->n, nt, TileTraits<C>::low,
                                              s->sem == QCS_CUDA_REFERENCE, RB)) {
    int rc = QCS_CUDA_OK;
    if (st.last - st.first == 1 || sweeps_cost_less(s, ops + st.first, st.last - st.first))
      for (int i = st.first; !rc && i < st.last; i++) rc = apply_op(s, ops[i]);
    else
      rc = launch_pass<C, RB>(s, ops, st);
    if (rc) return rc;
  }
  return QCS_CUDA_OK;
}

// Each quarter of an SM has an FP64 pipe of its own, which takes 64 cycles an
// instruction of a warp, and tiles of 64 threads leave half of them idle where
// an SM has one tile: a complex128 tile has 4 warps, of 8 amplitudes a thread,
// or of 4 with half the tile where that gives more SMs one.
// Sweeps of 4 layers of RY, RZ and a CNOT ladder, 16 amplitudes a thread against
// this: 12 qubits 337 -> 122 us, 16 (128 tiles of 2^9) 454 -> 177, 17 (128 of
// 2^10) 493 -> 308; from 18 qubits on an SM has two tiles and more,
// and 4 warps a tile still spread better (18, 20, 24 qubits, QFT and 200 gates,
// 16 amplitudes against 8: 701, 2166, 34748 us, 607, 1975, 34251).
// complex64 gates wait for their own latency where an SM has one or two tiles,
// which 8 warps of 8 amplitudes hide better than 4 of 16, and smaller tiles spread
// (300 random gates; 4, 8 amplitudes a thread in 2^10, 8 and 16 in 2^11): 13
// qubits 67, 71, 72, 83 us; 16 91, 95, 95, 115; 17 103, 100, 101, 120; 19 210,
// 143, 130, 147; 20 332, 230, 239, 192.  4 a thread gains little where it gains.
int run_tiles(qcs_cuda_state *s, const qcs_cuda_op *ops, int count) {
  const i64 sms = s->dev.num_sms;
  if (s->prec == QCS_CUDA_C64) {
    if (s->size >> 10 <= sms / 2) return run_tiles_t<float2, 3>(s, ops, count, 10);
    if (s->size >> 11 <= 2 * sms) return run_tiles_t<float2, 3>(s, ops, count, 11);
    return run_tiles_t<float2, 4>(s, ops, count, 11);
  }
  if (s->size >> 9 <= sms) return run_tiles_t<double2, 2>(s, ops, count, 9);
  return run_tiles_t<double2, 3>(s, ops, count, 10);
}

// A state smaller than one thread's registers stays with the sweeps.
bool tiles_supported(const qcs_cuda_state *s) { return s->n >= kTileRegBits; }

}  // namespace qcs

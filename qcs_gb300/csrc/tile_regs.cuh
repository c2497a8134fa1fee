// tile_regs.cuh -- a thread's amplitudes in registers, and the arithmetic of
// one-qubit gates on them, for the kernels that work on shared-memory tiles
// (tiles.cu, batch.cu).
//
// complex64 amplitudes are held two to a register pair: real parts of
// amplitudes 2u and 2u + 1 in one 64-bit register, imaginary parts in another,
// so that every product and sum is one packed FP32 instruction for two
// amplitudes and no instruction goes into exchanging parts.  Register bit 0
// (the "pair bit") tells the two apart: gates on the other bits combine whole
// registers, a gate on bit 0 combines a register with its halves exchanged.
// In shared memory real and imaginary parts lie apart too, so that any tile
// bit can be the pair bit.
//
// Rounding is that of the sweeps (cmul and cadd of common.cuh, as the compiler
// contracts them): a product of complex numbers is
//   (fma(d.x, v.x, -(d.y v.y)), fma(d.y, v.x, d.x v.y)),
// a sum of two products adds them after rounding.
#pragma once

#include <type_traits>

#include "common.cuh"

namespace qcs {

// ---- packed FP32 pairs -----------------------------------------------------
__device__ __forceinline__ u64 pack2(float lo, float hi) {
  u64 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ u64 both2(float s) { return pack2(s, s); }
// Products that add.rn.f32x2 sums are written a b + z with z = -0 that only the
// host knows.  Of a plain packed product and a packed sum the assembler makes
// one fused operation, with one rounding instead of two, .rn or not.

// Shared-memory position of tile amplitude i: its place in the 128-byte row
// is XORed with the row's number, so that whichever tile bits are held in
// registers a warp's lanes spread over the banks.  Linear over XOR.
// (complex64: of a real or imaginary part.)
__host__ __device__ __forceinline__ int tile_pos(int i, float2) {
  return i ^ ((i >> 5) & 31) ^ ((i >> 10) & 31);
}
__host__ __device__ __forceinline__ int tile_pos(int i, double2) {
  return i ^ ((i >> 3) & 7) ^ ((i >> 6) & 7) ^ ((i >> 9) & 7);
}

// One amplitude of a tile of L in shared memory.
__device__ __forceinline__ float2 tile_get(const float *S, int L, int at) {
  return make_float2(S[at], S[L + at]);
}
__device__ __forceinline__ void tile_put(float *S, int L, int at, float2 v) {
  S[at] = v.x;
  S[L + at] = v.y;
}
__device__ __forceinline__ double2 tile_get(const double2 *S, int, int at) { return S[at]; }
__device__ __forceinline__ void tile_put(double2 *S, int, int at, double2 v) { S[at] = v; }

// A gate's constants as packed operands: where the pair bit is the target (tb
// == 0) or a condition, the two halves take different ones.
//   dense  own and other entry's x, y, -y: (k0, k1, k2, k3) each for both
//          halves, or for tb == 0 (k0 | k3) then (k1 | k2)
//   diag   x, y, -y of k0, then of k1; for tb == 0 of (k0 | k1)
//   phase  x, y, -y of the phase; 1 + 0 i in the lower half under the pair bit
__device__ __forceinline__ void pack_factor(u64 *c, float xl, float yl, float xh, float yh) {
  c[0] = pack2(xl, xh);
  c[1] = pack2(yl, yh);
  c[2] = pack2(-yl, -yh);
}
__device__ __forceinline__ void pack_dense(u64 *c, int tb, const float *k) {
  if (tb == 0) {
    pack_factor(c, k[0], k[1], k[6], k[7]);
    pack_factor(c + 3, k[2], k[3], k[4], k[5]);
  } else {
#pragma unroll
    for (int e = 0; e < 4; e++) pack_factor(c + 3 * e, k[2 * e], k[2 * e + 1], k[2 * e], k[2 * e + 1]);
  }
}
__device__ __forceinline__ void pack_diag(u64 *c, int tb, const float *k) {
  if (tb == 0) {
    pack_factor(c, k[0], k[1], k[2], k[3]);
  } else {
    pack_factor(c, k[0], k[1], k[0], k[1]);
    pack_factor(c + 3, k[2], k[3], k[2], k[3]);
  }
}
__device__ __forceinline__ void pack_phase(u64 *c, int cond, const float *k) {
  const bool p = cond & 1;
  pack_factor(c, p ? 1.f : k[0], p ? 0.f : k[1], k[0], k[1]);
}

// f(0), f(1), ... f(N - 1), the argument a constant.
template <int N, int I = 0, typename F>
__device__ __forceinline__ void each(F &&f) {
  if constexpr (I < N) {
    f(std::integral_constant<int, I>());
    each<N, I + 1>(f);
  }
}

// 2^RB amplitudes of a complex64 tile.  S: 2^nt real parts, then 2^nt
// imaginary parts.
//
// The amplitudes are PTX registers qre<u>, qim<u>, declared once in the kernel
// that uses them and updated in place by name.  As C++ variables they pass
// through the merge of the gate dispatch's branches, and there the compiler
// moved every one of them for every gate: 117 of the 300 instructions an
// amplitude took in a pass of 37 gates (157M -> 109M instructions at 24 qubits).
#define QCS_REGS_F32_DECLARE(N) \
  asm volatile(".reg .b64 qre<%0>;\n.reg .b64 qim<%0>;" ::"n"(N))
template <int RB> struct RegsF32 {
  static constexpr int N = 1 << RB, U = N / 2;
  typedef float R;

  __device__ __forceinline__ void load(const float *S, int L, const int (&pos)[N]) {
    each<U>([&](auto uc) {
      constexpr int u = decltype(uc)::value;
      asm volatile("mov.b64 qre%0, {%1, %2};\nmov.b64 qim%0, {%3, %4};" ::"n"(u),
                   "f"(S[pos[2 * u]]), "f"(S[pos[2 * u + 1]]), "f"(S[L + pos[2 * u]]),
                   "f"(S[L + pos[2 * u + 1]]));
    });
  }
  __device__ __forceinline__ void store(float *S, int L, const int (&pos)[N]) const {
    each<U>([&](auto uc) {
      constexpr int u = decltype(uc)::value;
      float a, b, c, d;
      asm volatile("mov.b64 {%0, %1}, qre%4;\nmov.b64 {%2, %3}, qim%4;"
                   : "=f"(a), "=f"(b), "=f"(c), "=f"(d) : "n"(u));
      S[pos[2 * u]] = a;
      S[pos[2 * u + 1]] = b;
      S[L + pos[2 * u]] = c;
      S[L + pos[2 * u + 1]] = d;
    });
  }

  // The same; whether an amplitude is an infinity or a NaN: 0 x is a NaN for those
  // alone.
  __device__ __forceinline__ bool store_finite(float *S, int L, const int (&pos)[N]) const {
    float z[4] = {0.f, 0.f, 0.f, 0.f};  // as many chains
    each<U>([&](auto uc) {
      constexpr int u = decltype(uc)::value;
      float a, b, c, d;
      asm volatile("mov.b64 {%0, %1}, qre%4;\nmov.b64 {%2, %3}, qim%4;"
                   : "=f"(a), "=f"(b), "=f"(c), "=f"(d) : "n"(u));
      S[pos[2 * u]] = a;
      S[pos[2 * u + 1]] = b;
      S[L + pos[2 * u]] = c;
      S[L + pos[2 * u + 1]] = d;
      z[0] = fmaf(a, 0.f, z[0]);
      z[1] = fmaf(b, 0.f, z[1]);
      z[2] = fmaf(c, 0.f, z[2]);
      z[3] = fmaf(d, 0.f, z[3]);
    });
    return (z[0] + z[1]) + (z[2] + z[3]) != 0.f;
  }

  // f(u, w) for the register pairs that differ in register bit TB >= 1
  template <int TB, typename F>
  static __device__ __forceinline__ void pairs(F &&f) {
    each<U>([&](auto uc) {
      constexpr int u = decltype(uc)::value;
      if constexpr (!(u & (1 << (TB - 1))))
        f(uc, std::integral_constant<int, u | (1 << (TB - 1))>());
    });
  }

  // k = a, b, c, d: [[a, b], [c, d]], all real, on register bit TB: two rounded products, then
  // their sum.
  template <int TB>
  __device__ __forceinline__ void real(const float *k, u64 z) {
    if constexpr (TB == 0) {
      const u64 ad = pack2(k[0], k[3]), bc = pack2(k[1], k[2]);
      each<U>([&](auto uc) {
        constexpr int u = decltype(uc)::value;
        asm volatile(
            "{\n.reg .b32 l, h;\n.reg .b64 s;\n"
            "mov.b64 {l, h}, qre%0;\nmov.b64 s, {h, l};\n"
            "fma.rn.f32x2 s, %2, s, %3;\nfma.rn.f32x2 qre%0, %1, qre%0, %3;\n"
            "add.rn.f32x2 qre%0, qre%0, s;\n"
            "mov.b64 {l, h}, qim%0;\nmov.b64 s, {h, l};\n"
            "fma.rn.f32x2 s, %2, s, %3;\nfma.rn.f32x2 qim%0, %1, qim%0, %3;\n"
            "add.rn.f32x2 qim%0, qim%0, s;\n}" ::"n"(u), "l"(ad), "l"(bc), "l"(z));
      });
    } else {
      const u64 aa = both2(k[0]), bb = both2(k[1]), cc = both2(k[2]), dd = both2(k[3]);
      pairs<TB>([&](auto uc, auto wc) {
        constexpr int u = decltype(uc)::value, w = decltype(wc)::value;
        asm volatile(
            "{\n.reg .b64 s, t;\n"
            "fma.rn.f32x2 s, %3, qre%1, %6;\nfma.rn.f32x2 qre%1, %5, qre%1, %6;\n"
            "fma.rn.f32x2 t, %4, qre%0, %6;\nfma.rn.f32x2 qre%0, %2, qre%0, %6;\n"
            "add.rn.f32x2 qre%0, qre%0, s;\nadd.rn.f32x2 qre%1, qre%1, t;\n"
            "fma.rn.f32x2 s, %3, qim%1, %6;\nfma.rn.f32x2 qim%1, %5, qim%1, %6;\n"
            "fma.rn.f32x2 t, %4, qim%0, %6;\nfma.rn.f32x2 qim%0, %2, qim%0, %6;\n"
            "add.rn.f32x2 qim%0, qim%0, s;\nadd.rn.f32x2 qim%1, qim%1, t;\n}" ::"n"(u),
            "n"(w), "l"(aa), "l"(bb), "l"(cc), "l"(dd), "l"(z));
      });
    }
  }

  // A 2x2 with the four complex entries k on register bit TB.
  template <int TB>
  __device__ __forceinline__ void dense(const float *f) {
    u64 k[12];
    pack_dense(k, TB, f);
    if constexpr (TB == 0) {
      const u64 ax = k[0], ay = k[1], an = k[2], bx = k[3], by = k[4], bn = k[5];
      each<U>([&](auto uc) {
        constexpr int u = decltype(uc)::value;
        asm volatile(
            "{\n.reg .b32 l, h;\n.reg .b64 r, i, s, t, v;\n"
            "mov.b64 {l, h}, qre%0;\nmov.b64 r, {h, l};\n"
            "mov.b64 {l, h}, qim%0;\nmov.b64 i, {h, l};\n"
            "mul.rn.f32x2 s, %3, qim%0;\nfma.rn.f32x2 s, %1, qre%0, s;\n"
            "mul.rn.f32x2 t, %1, qim%0;\nfma.rn.f32x2 t, %2, qre%0, t;\n"
            "mul.rn.f32x2 v, %6, i;\nfma.rn.f32x2 v, %4, r, v;\nadd.rn.f32x2 qre%0, s, v;\n"
            "mul.rn.f32x2 v, %4, i;\nfma.rn.f32x2 v, %5, r, v;\nadd.rn.f32x2 qim%0, t, v;\n}"
            ::"n"(u), "l"(ax), "l"(ay), "l"(an), "l"(bx), "l"(by), "l"(bn));
      });
    } else {
      const u64 ax = k[0], ay = k[1], an = k[2], bx = k[3], by = k[4], bn = k[5];
      const u64 cx = k[6], cy = k[7], cn = k[8], dx = k[9], dy = k[10], dn = k[11];
      pairs<TB>([&](auto uc, auto wc) {
        constexpr int u = decltype(uc)::value, w = decltype(wc)::value;
        asm volatile(
            "{\n.reg .b64 s, t, v, x;\n"
            "mul.rn.f32x2 s, %4, qim%0;\nfma.rn.f32x2 s, %2, qre%0, s;\n"
            "mul.rn.f32x2 t, %2, qim%0;\nfma.rn.f32x2 t, %3, qre%0, t;\n"
            "mul.rn.f32x2 v, %7, qim%1;\nfma.rn.f32x2 v, %5, qre%1, v;\nadd.rn.f32x2 s, s, v;\n"
            "mul.rn.f32x2 v, %5, qim%1;\nfma.rn.f32x2 v, %6, qre%1, v;\nadd.rn.f32x2 t, t, v;\n"
            "mul.rn.f32x2 v, %10, qim%0;\nfma.rn.f32x2 v, %8, qre%0, v;\n"
            "mul.rn.f32x2 x, %8, qim%0;\nfma.rn.f32x2 x, %9, qre%0, x;\n"
            "mov.b64 qre%0, s;\nmov.b64 qim%0, t;\n"
            "mul.rn.f32x2 s, %13, qim%1;\nfma.rn.f32x2 s, %11, qre%1, s;\n"
            "mul.rn.f32x2 t, %11, qim%1;\nfma.rn.f32x2 t, %12, qre%1, t;\n"
            "add.rn.f32x2 qre%1, v, s;\nadd.rn.f32x2 qim%1, x, t;\n}" ::"n"(u), "n"(w), "l"(ax),
            "l"(ay), "l"(an), "l"(bx), "l"(by), "l"(bn), "l"(cx), "l"(cy), "l"(cn), "l"(dx),
            "l"(dy), "l"(dn));
      });
    }
  }

  // X on register bit TB, where register bit CB (-1: none) is set
  template <int TB, int CB>
  __device__ __forceinline__ void exchange() {
    static_assert(TB != CB, "control equals target");
    if constexpr (TB == 0) {
      each<U>([&](auto uc) {
        constexpr int u = decltype(uc)::value;
        if constexpr (CB < 0 || (u >> (CB < 1 ? 0 : CB - 1)) & 1)
          asm volatile("{\n.reg .b32 l, h;\nmov.b64 {l, h}, qre%0;\nmov.b64 qre%0, {h, l};\n"
                       "mov.b64 {l, h}, qim%0;\nmov.b64 qim%0, {h, l};\n}" ::"n"(u));
      });
    } else {
      pairs<TB>([&](auto uc, auto wc) {
        constexpr int u = decltype(uc)::value, w = decltype(wc)::value;
        if constexpr (CB == 0)  // the upper halves
          asm volatile("{\n.reg .b32 a, b, c, d;\n"
                       "mov.b64 {a, b}, qre%0;\nmov.b64 {c, d}, qre%1;\n"
                       "mov.b64 qre%0, {a, d};\nmov.b64 qre%1, {c, b};\n"
                       "mov.b64 {a, b}, qim%0;\nmov.b64 {c, d}, qim%1;\n"
                       "mov.b64 qim%0, {a, d};\nmov.b64 qim%1, {c, b};\n}" ::"n"(u), "n"(w));
        else if constexpr (CB < 0 || (u >> (CB < 1 ? 0 : CB - 1)) & 1)
          asm volatile("{\n.reg .b64 s;\nmov.b64 s, qre%0;\nmov.b64 qre%0, qre%1;\n"
                       "mov.b64 qre%1, s;\nmov.b64 s, qim%0;\nmov.b64 qim%0, qim%1;\n"
                       "mov.b64 qim%1, s;\n}" ::"n"(u), "n"(w));
      });
    }
  }

  // The phase f0 + i f1 where the register bits `cond` are set.
  __device__ __forceinline__ void phase_where(const float *f, int cond) {
    u64 k[3];
    pack_phase(k, cond, f);
    const u64 xx = k[0], yy = k[1], ny = k[2];
    each<U>([&](auto uc) {
      constexpr int u = decltype(uc)::value;
      if ((u & (cond >> 1)) == (cond >> 1)) turn<u>(xx, yy, ny);
    });
  }

  // k = c, s: [[c, i s], [i s, c]]
  template <int TB>
  __device__ __forceinline__ void rx(const float *k, u64 z) {
    const u64 cc = both2(k[0]), ss = both2(k[1]), ns = both2(-k[1]);
    if constexpr (TB == 0) {
      each<U>([&](auto uc) {
        constexpr int u = decltype(uc)::value;
        asm volatile(
            "{\n.reg .b32 l, h;\n.reg .b64 s, t;\n"
            "mov.b64 {l, h}, qre%0;\nmov.b64 s, {h, l};\n"
            "mov.b64 {l, h}, qim%0;\nmov.b64 t, {h, l};\n"
            "fma.rn.f32x2 s, %2, s, %4;\nfma.rn.f32x2 t, %3, t, %4;\n"
            "fma.rn.f32x2 qre%0, %1, qre%0, %4;\nfma.rn.f32x2 qim%0, %1, qim%0, %4;\n"
            "add.rn.f32x2 qre%0, qre%0, t;\nadd.rn.f32x2 qim%0, qim%0, s;\n}" ::"n"(u),
            "l"(cc), "l"(ss), "l"(ns), "l"(z));
      });
    } else {
      pairs<TB>([&](auto uc, auto wc) {
        constexpr int u = decltype(uc)::value, w = decltype(wc)::value;
        asm volatile(
            "{\n.reg .b64 s, t;\n"
            "fma.rn.f32x2 s, %4, qim%1, %5;\nfma.rn.f32x2 t, %3, qre%0, %5;\n"
            "fma.rn.f32x2 qre%0, %2, qre%0, %5;\nfma.rn.f32x2 qim%1, %2, qim%1, %5;\n"
            "add.rn.f32x2 qre%0, qre%0, s;\nadd.rn.f32x2 qim%1, qim%1, t;\n"
            "fma.rn.f32x2 s, %4, qim%0, %5;\nfma.rn.f32x2 t, %3, qre%1, %5;\n"
            "fma.rn.f32x2 qre%1, %2, qre%1, %5;\nfma.rn.f32x2 qim%0, %2, qim%0, %5;\n"
            "add.rn.f32x2 qre%1, qre%1, s;\nadd.rn.f32x2 qim%0, qim%0, t;\n}" ::"n"(u),
            "n"(w), "l"(cc), "l"(ss), "l"(ns), "l"(z));
      });
    }
  }

  // Y: v0' = -i v1, v1' = i v0
  template <int TB>
  __device__ __forceinline__ void y() {
    if constexpr (TB == 0) {
      each<U>([&](auto uc) {
        constexpr int u = decltype(uc)::value;
        asm volatile(
            "{\n.reg .b32 a, b, c, d;\n"
            "mov.b64 {a, b}, qre%0;\nmov.b64 {c, d}, qim%0;\n"
            "xor.b32 c, c, 0x80000000;\nxor.b32 b, b, 0x80000000;\n"
            "mov.b64 qre%0, {d, c};\nmov.b64 qim%0, {b, a};\n}" ::"n"(u));
      });
    } else {
      pairs<TB>([&](auto uc, auto wc) {
        constexpr int u = decltype(uc)::value, w = decltype(wc)::value;
        asm volatile(
            "{\n.reg .b64 s, t;\nmov.b64 s, qre%0;\nmov.b64 t, qim%0;\n"
            "mov.b64 qre%0, qim%1;\nxor.b64 qim%0, qre%1, 0x8000000080000000;\n"
            "xor.b64 qre%1, t, 0x8000000080000000;\nmov.b64 qim%1, s;\n}" ::"n"(u), "n"(w));
      });
    }
  }

  // The complex factor (x, y) on register u; halves apart.
  template <int u>
  static __device__ __forceinline__ void turn(u64 x, u64 y, u64 ny) {
    asm volatile(
        "{\n.reg .b64 s, t;\n"
        "mul.rn.f32x2 s, %3, qim%0;\nmul.rn.f32x2 t, %1, qim%0;\n"
        "fma.rn.f32x2 qim%0, %2, qre%0, t;\nfma.rn.f32x2 qre%0, %1, qre%0, s;\n}" ::"n"(u),
        "l"(x), "l"(y), "l"(ny));
  }

  // diag(k0 + i k1, k2 + i k3) on register bit TB
  template <int TB>
  __device__ __forceinline__ void diag(const float *f) {
    u64 k[6];
    pack_diag(k, TB, f);
    if constexpr (TB == 0) {
      const u64 x = k[0], y = k[1], ny = k[2];
      each<U>([&](auto uc) { turn<decltype(uc)::value>(x, y, ny); });
    } else {
      const u64 x0 = k[0], y0 = k[1], n0 = k[2], x1 = k[3], y1 = k[4], n1 = k[5];
      pairs<TB>([&](auto uc, auto wc) {
        turn<decltype(uc)::value>(x0, y0, n0);
        turn<decltype(wc)::value>(x1, y1, n1);
      });
    }
  }

  // k0 + i k1 on every amplitude whose register bits COND are set.  With the
  // pair bit among them, the other half takes the factor 1 + 0 i.
  template <int COND>
  __device__ __forceinline__ void phase(const float *f) {
    u64 k[3];
    pack_phase(k, COND, f);
    const u64 xx = k[0], yy = k[1], ny = k[2];
    each<U>([&](auto uc) {
      constexpr int u = decltype(uc)::value;
      if constexpr ((u & (COND >> 1)) == (COND >> 1)) turn<u>(xx, yy, ny);
    });
  }

  // -1 on every amplitude whose register bits `cond` are set
  __device__ __forceinline__ void sign(int cond) {
    const u64 flip = (0x80000000ull << 32) | ((cond & 1) ? 0ull : 0x80000000ull);
    each<U>([&](auto uc) {
      constexpr int u = decltype(uc)::value;
      if ((u & (cond >> 1)) == (cond >> 1))
        asm volatile("xor.b64 qre%0, qre%0, %1;\nxor.b64 qim%0, qim%0, %1;" ::"n"(u),
                     "l"(flip));
    });
  }

  // v0 := v1 where the register bits `cond` are set
  template <int TB>
  __device__ __forceinline__ void copy(int cond) {
    if constexpr (TB == 0) {
      each<U>([&](auto uc) {
        constexpr int u = decltype(uc)::value;
        if ((u & (cond >> 1)) == (cond >> 1))
          asm volatile("{\n.reg .b32 l, h;\nmov.b64 {l, h}, qre%0;\nmov.b64 qre%0, {h, h};\n"
                       "mov.b64 {l, h}, qim%0;\nmov.b64 qim%0, {h, h};\n}" ::"n"(u));
      });
    } else {
      // the low halves too, unless the pair bit is a condition
      const u64 take = (0xffffffffull << 32) | ((cond & 1) ? 0ull : 0xffffffffull);
      pairs<TB>([&](auto uc, auto wc) {
        constexpr int u = decltype(uc)::value, w = decltype(wc)::value;
        if ((u & (cond >> 1)) == (cond >> 1))
          asm volatile(
              "{\n.reg .b64 s;\n"
              "xor.b64 s, qre%0, qre%1;\nand.b64 s, s, %2;\nxor.b64 qre%0, qre%0, s;\n"
              "xor.b64 s, qim%0, qim%1;\nand.b64 s, s, %2;\nxor.b64 qim%0, qim%0, s;\n}"
              ::"n"(u), "n"(w), "l"(take));
      });
    }
  }
};

// 2^RB amplitudes of a complex128 tile (re, im interleaved in shared memory).
// The FP64 pipe bounds this one, not the instruction count.
template <int RB> struct RegsF64 {
  static constexpr int N = 1 << RB;
  typedef double R;
  double2 a[N];

  __device__ __forceinline__ void load(const double2 *S, int, const int (&pos)[N]) {
#pragma unroll
    for (int e = 0; e < N; e++) a[e] = S[pos[e]];
  }
  __device__ __forceinline__ void store(double2 *S, int, const int (&pos)[N]) const {
#pragma unroll
    for (int e = 0; e < N; e++) S[pos[e]] = a[e];
  }
  static __device__ __forceinline__ double2 scale(double s, double2 v) {
    return make_double2(__dmul_rn(s, v.x), __dmul_rn(s, v.y));
  }
  template <int TB>
  __device__ __forceinline__ void real(const double *k, u64) {
    const double p = k[0], q = k[1], r = k[2], s = k[3];
#pragma unroll
    for (int e = 0; e < N; e++) {
      if (e & (1 << TB)) continue;
      const int f = e | (1 << TB);
      const double2 v0 = a[e], v1 = a[f];
      a[e] = cadd(scale(p, v0), scale(q, v1));
      a[f] = cadd(scale(r, v0), scale(s, v1));
    }
  }
  // k0 * [[1, 1], [1, -1]]: the products serve both outputs
  template <int TB>
  __device__ __forceinline__ void had(const double *k) {
    const double h = k[0];
#pragma unroll
    for (int e = 0; e < N; e++) {
      if (e & (1 << TB)) continue;
      const int f = e | (1 << TB);
      const double2 x0 = scale(h, a[e]), x1 = scale(h, a[f]);
      a[e] = cadd(x0, x1);
      a[f] = make_double2(__dsub_rn(x0.x, x1.x), __dsub_rn(x0.y, x1.y));
    }
  }
  template <int TB>
  __device__ __forceinline__ void rx(const double *k, u64) {
    const double c = k[0], s = k[1];
#pragma unroll
    for (int e = 0; e < N; e++) {
      if (e & (1 << TB)) continue;
      const int f = e | (1 << TB);
      const double2 v0 = a[e], v1 = a[f];
      a[e].x = __dsub_rn(__dmul_rn(c, v0.x), __dmul_rn(s, v1.y));
      a[e].y = __dadd_rn(__dmul_rn(c, v0.y), __dmul_rn(s, v1.x));
      a[f].x = __dsub_rn(__dmul_rn(c, v1.x), __dmul_rn(s, v0.y));
      a[f].y = __dadd_rn(__dmul_rn(c, v1.y), __dmul_rn(s, v0.x));
    }
  }
  template <int TB>
  __device__ __forceinline__ void y() {
#pragma unroll
    for (int e = 0; e < N; e++) {
      if (e & (1 << TB)) continue;
      const int f = e | (1 << TB);
      const double2 v0 = a[e], v1 = a[f];
      a[e] = make_double2(v1.y, -v1.x);
      a[f] = make_double2(-v0.y, v0.x);
    }
  }
  template <int TB>
  __device__ __forceinline__ void diag(const double *k) {
    const double2 d0 = make_double2(k[0], k[1]), d1 = make_double2(k[2], k[3]);
#pragma unroll
    for (int e = 0; e < N; e++) a[e] = cmul((e & (1 << TB)) ? d1 : d0, a[e]);
  }
  // COND is static: a product that is only predicated off would still take
  // its slot in the FP64 pipe.
  template <int COND>
  __device__ __forceinline__ void phase(const double *k) {
    const double2 d = make_double2(k[0], k[1]);
#pragma unroll
    for (int e = 0; e < N; e++)
      if ((e & COND) == COND) a[e] = cmul(d, a[e]);
  }
  __device__ __forceinline__ void sign(int cond) {
#pragma unroll
    for (int e = 0; e < N; e++)
      if ((e & cond) == cond) a[e] = make_double2(-a[e].x, -a[e].y);
  }
  template <int TB>
  __device__ __forceinline__ void copy(int cond) {
#pragma unroll
    for (int e = 0; e < N; e++) {
      if (e & (1 << TB)) continue;
      if ((e & cond) == cond) a[e] = a[e | (1 << TB)];
    }
  }
};

}  // namespace qcs

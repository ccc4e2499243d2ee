// Symmetric eigenproblems and dense products of one molecule in 64-bit
// accuracy on the 16-bit tensor instructions, by a TEAM of CTAs (linalg.cuh).
//
// The FP64 pipe of this part issues 1.7 FMA per clock and SM, the 16-bit
// tensor instruction (mma.sync m16n8k16) 1020 (both measured): a product of
// 60-bit fixed-point operands cut into six digits of ten bits takes 21 digit
// products (orders p + q <= 5), still ~28 times the FP64 rate (error-free
// splitting as in Ozaki, Ogita, Oishi and Rump, Numer. Algorithms 59 (2012) 95,
// with a fixed cut). The orders left out are 2^-64 sqrt(5 n) of the operands'
// norms. The digit product sums are integers in float32 accumulators, exact below
// 2^24 and rounded to an integer above. Six digits: the orders 0 to 2 are exact
// for any operands of norm <= 1 (order 2 is carried upwards every 32 terms, all
// orders every 64); from order 3 on, of weight <= 2^-50, for digits that are not
// all at their limit. Three digits: orders 0 and 1 are exact for operands of norm
// <= 1, order 2 can reach 4.5e7 in its 128 terms and is then rounded to a multiple
// of 4, 2^-38 of operands that are cut at 2^-31. An update's left operand E^T
// has rows of norm <= 8 and V columns of norm < 2, so that its values stay below
// 16 as everywhere (2^24 in order 0, tile_fix); its order 1 may round the same
// way, which the next step's R and T see, and which is below 2^-53 in the last
// step, where E < 2^-28.
// Nine-bit digits (54 bits) lost 2^-58 sqrt(5 n), with a sign on a diagonal: SCF
// residuals then end at 6e-12 (n = 181) to 6e-10 (n = 1145), where float64 ends
// at 6e-13 to 4e-12.
//
// Fixed point: an operand's value is sum_p digit_p 2^(-10 (p + 1)) times a
// power of two kept beside the matrix (per matrix or per row); digits are
// balanced (|digit| <= 512) but the first, which takes the rest (|.| <= 2048,
// exact in fp16, so |value| <= 2). Results are 64-bit integers of weight 2^-58.
//
// Digit planes are stored in the register layout of the instruction: a block
// of 16 x 16 values is one 16-byte word per lane and plane. The four registers
// of an A operand (rows i, inner index k) in the order 0, 2, 1, 3 are those of
// two B operands (C = A B^T), so a matrix is stored in the order of the side
// it stands on ("left" or "right") and no register is moved between a load and
// the instruction; X and V stand on both and are stored for the left only (a
// second copy cost more in L2 misses than the moves). A result tile has the
// layout of an A operand, transposed blocks come from movmatrix.
//
// Eigenvectors are iterated (Ogita and Aishima, Japan J. Indust. Appl. Math.
// 35 (2018) 1007, here with the first-order rotation clamped): for approximate
// vectors in the rows of V, T = V F V^T and R = I - V V^T give
//   lam_i = T_ii / (1 - R_ii),
//   Z_ij = (T_ij + (lam_i + lam_j) R_ij / 2) / (lam_j - lam_i),
//   V <- V + (R / 2 + Z)^T V,
// which converges quadratically and needs only products. Steps far from
// convergence take three digits (6 digit products instead of 21). The vectors
// of one SCF iteration start those of the next.
//
// Measured against the Householder / float64 path (GB300, energy + forces):
// one molecule of 72 orbitals 36.9 -> 8.0 ms, of 233 orbitals 292 -> 28.4 ms
// (there 4 CTAs, here 16), 256 molecules of 22-172 orbitals 223 -> 71.7 ms, with
// no larger distance from the CPU oracle over the benchmark sets (|dE| <= 7.0e-12
// Eh, |dF| <= 5.2e-12 Eh/Bohr; 7.0e-12 and 1.2e-10 there).
#pragma once
#include <cuda_fp16.h>

#include "linalg.cuh"

namespace dxtb {

constexpr int kDig = 6;          // digits of a full operand
constexpr int kDigLow = 3;       // digits of the coarse steps and of the rotations
constexpr int kW = 60, kR = 58;  // an operand's last digit weighs 2^-kW, results 2^-kR
constexpr int kMaxSteps = 160;   // steps of one eigenproblem before it is given up
constexpr float kZMax = 0.4f;    // largest rotation of one pair in one step
constexpr float kZNorm = 1.2f;   // largest Frobenius norm (over sqrt 2) of the rotations of a small problem
constexpr float kFinal = 0x1p-28f;   // a full step of this Frobenius norm is the last (its error is quadratic)
constexpr float kZLow = 0x1p-7f;    // above this the next step is coarse

__host__ __device__ inline int64_t blocks16(int64_t n) { return (n + 15) / 16; }

__device__ __forceinline__ void mma16816(float *c, const uint4 &a, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3},{%4,%5,%6,%7},{%8,%9},{%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1));
}

// A word of planes. Other warps write them in earlier phases: not the
// read-only path, and volatile so that no load moves across a barrier.
__device__ __forceinline__ uint4 ld_plane(const uint4 *p) {
  uint4 v;
  asm volatile("ld.global.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(__cvta_generic_to_global(p)));
  return v;
}
// A word read once per pass over data that exceeds the caches (the integrals,
// 80 bytes a pair): kept out of the L1 and first to leave the L2, where the
// planes of the running steps should stay.
__device__ __forceinline__ uint64_t stream_policy() {
  uint64_t pol;
  asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
  return pol;
}
__device__ __forceinline__ int4 ld_stream(const int4 *p, uint64_t pol) {
  int4 v;
  asm volatile("ld.global.L1::no_allocate.L2::cache_hint.v4.s32 {%0,%1,%2,%3}, [%4], %5;"
      : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
      : "l"(__cvta_generic_to_global(p)), "l"(pol));
  return v;
}
__device__ __forceinline__ void st_plane(uint4 *p, const uint4 &v) {
  asm volatile("st.global.v4.u32 [%0], {%1,%2,%3,%4};" ::"l"(__cvta_generic_to_global(p)), "r"(v.x), "r"(v.y),
               "r"(v.z), "r"(v.w)
               : "memory");
}

// The 16 x 16 tile sum_k A[i][k] B[j][k] over the k blocks [k0, k1) with NP
// digits, as the sums of each order (acc[d], weight 2^(-10 (d + 2)), integers):
// A, B are the first blocks of the two block rows, sa, sb the words
// per block (planes stored x 32). Value e: row g + 8 ((e >> 1) & 1), column
// 8 (e >> 2) + 2 q + (e & 1) for lane 4 g + q. Orders are carried into the one
// above (multiples of 1024); what stays exact is said at the top.
template <int NP>
__device__ __forceinline__ void tile_nt(const uint4 *A, int sa, const uint4 *B, int sb, bool left_b, int k0, int k1,
                                        float (&acc)[NP][8]) {
  const int lane = threadIdx.x & 31;
  const uint4 *pa = A + (size_t)k0 * sa + lane, *pb = B + (size_t)k0 * sb + lane;
#pragma unroll
  for (int p = 0; p < NP; ++p)
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[p][e] = 0.0f;
  constexpr int kDrain = NP == kDigLow ? 8 : 4;  // k blocks of 16 between carries of all orders
  int left = kDrain;
  constexpr int kUnroll = NP == kDigLow ? 2 : 1;  // loads of two k blocks in flight where registers allow
#pragma unroll kUnroll
  for (int kb = k0; kb < k1; ++kb) {
    uint4 a[NP];
#pragma unroll
    for (int p = 0; p < NP; ++p) a[p] = ld_plane(pa + p * 32);
#pragma unroll
    for (int q = 0; q < NP; ++q) {
      uint4 b = ld_plane(pb + q * 32);
      if (left_b) {  // the order of the left side: swap the middle words
        const uint32_t y = b.y;
        b.y = b.z;
        b.z = y;
      }
#pragma unroll
      for (int p = 0; p < NP - q; ++p) {
        mma16816(acc[p + q], a[p], b.x, b.y);
        mma16816(acc[p + q] + 4, a[p], b.z, b.w);
      }
    }
    pa += sa;
    pb += sb;
    auto carry = [&](int p) {
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float c = fmaf(acc[p][e], 0x1p-10f, 0x1.8p23f) - 0x1.8p23f;  // rounded to an integer
        acc[p - 1][e] += c;
        acc[p][e] = fmaf(-1024.0f, c, acc[p][e]);
      }
    };
    if (--left == 0) {
      left = kDrain;
      if (kb + 1 < k1) {
#pragma unroll
        for (int p = NP - 1; p > 0; --p) carry(p);
      }
    } else if (NP == kDig && left == 2) {
      carry(2);
    }
  }
}

// an integer in float32 (|x| < 2^22) as an int: no conversion (those run at
// an eighth of the rate)
__device__ __forceinline__ int int_f(float x) { return __float_as_int(x + 0x1.8p23f) - 0x4b400000; }

// A tile's value e less one (where asked) in float32: where the leading orders
// cancel the partial results are exact integers, so the error is relative.
template <int NP>
__device__ __forceinline__ float tile_float(const float (&acc)[NP][8], int e, bool less_one) {
  float v = less_one ? acc[0][e] - 0x1p20f : acc[0][e];
#pragma unroll
  for (int p = 1; p < NP; ++p) v = fmaf(v, 1024.0f, acc[p][e]);
  return v * (NP == 6 ? 0x1p-70f : 0x1p-40f);
}

// A tile's value e as the NP digits of an operand, and the rest below the last
// (weight 2^(-10 (NP + 1)), |rest| <= 512). Carries in float32, all exact.
template <int NP>
__device__ __forceinline__ float tile_digits(const float (&acc)[NP][8], int e, float (&d)[NP]) {
  float c = fmaf(acc[NP - 1][e], 0x1p-10f, 0x1.8p23f) - 0x1.8p23f;
  const float rest = fmaf(-1024.0f, c, acc[NP - 1][e]);
#pragma unroll
  for (int i = NP - 1; i > 0; --i) {
    const float x = acc[i - 1][e] + c;
    c = fmaf(x, 0x1p-10f, 0x1.8p23f) - 0x1.8p23f;
    d[i] = fmaf(-1024.0f, c, x);
  }
  d[0] = c;
  return rest;
}

// A tile's value e as an integer of weight 2^-kR (|value| < 16).
template <int NP>
__device__ __forceinline__ long long tile_fix(const float (&acc)[NP][8], int e) {
  float d[NP];
  const float rest = tile_digits<NP>(acc, e, d);
  const long long hi = (long long)int_f(d[0]) * (1 << 20) + (int_f(d[1]) * 1024 + int_f(d[2]));  // weight 2^-30
  if constexpr (NP > 3) {
    const int lo = (int_f(d[3]) * 1024 + int_f(d[4])) * 1024 + int_f(d[5]);  // weight 2^-60
    return hi * (1 << 28) + ((lo + 2) >> 2);
  } else {
    return hi * (1 << 28) + int_f(rest) * (1 << 18);
  }
}

// Balanced digits of r (weight 2^-kW, |r| < 2^61), first digit first. With NP = 3
// the value is rounded to 2^-30, which leaves the first three digits of NP = 6.
template <int NP>
__device__ __forceinline__ void cut(long long r, int (&d)[NP]) {
  const int hi = (int)((r + (1 << 29)) >> 30);
  if constexpr (NP == 6) {
    const int lo = (int)(r - ((long long)hi << 30));
    const int x1 = (lo + 512) >> 10, x2 = (x1 + 512) >> 10;
    d[5] = lo - (x1 << 10);
    d[4] = x1 - (x2 << 10);
    d[3] = x2;
  }
  const int y1 = (hi + 512) >> 10, y2 = (y1 + 512) >> 10;
  d[2] = hi - (y1 << 10);
  d[1] = y1 - (y2 << 10);
  d[0] = y2;
}

// Two digits as fp16. |d| <= 512: the bits of 1536 + d (unit spacing there)
// minus 1536; the first digit by conversion.
__device__ __forceinline__ uint32_t pack_small(int a, int b) {
  const uint32_t w = (uint32_t)(a + 0x6600) | ((uint32_t)(b + 0x6600) << 16);
  const __half2 h = __hsub2(*reinterpret_cast<const __half2 *>(&w), __half2half2(__ushort_as_half(0x6600)));
  return *reinterpret_cast<const uint32_t *>(&h);
}
__device__ __forceinline__ uint32_t pack_first(int a, int b) {
  const __half2 h = __floats2half2_rn((float)a, (float)b);
  return *reinterpret_cast<const uint32_t *>(&h);
}

// Digit words of one block: value e of the lane (tile_nt's order) as r[e].
template <int NP>
__device__ __forceinline__ void cut_block(const long long (&r)[8], uint32_t (&w)[NP][4]) {
#pragma unroll
  for (int h = 0; h < 4; ++h) {
    int a[NP], b[NP];
    cut<NP>(r[2 * h], a);
    cut<NP>(r[2 * h + 1], b);
    w[0][h] = pack_first(a[0], b[0]);
#pragma unroll
    for (int p = 1; p < NP; ++p) w[p][h] = pack_small(a[p], b[p]);
  }
}

// Digit words of values of weight 2^-30.
__device__ __forceinline__ void cut_words(const int (&r)[8], uint32_t (&w)[kDigLow][4]) {
#pragma unroll
  for (int h = 0; h < 4; ++h) {
    int d[2][3];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int x = r[2 * h + k], y1 = (x + 512) >> 10, y2 = (y1 + 512) >> 10;
      d[k][2] = x - (y1 << 10);
      d[k][1] = y1 - (y2 << 10);
      d[k][0] = y2;
    }
    w[0][h] = pack_first(d[0][0], d[1][0]);
    w[1][h] = pack_small(d[0][1], d[1][1]);
    w[2][h] = pack_small(d[0][2], d[1][2]);
  }
}

// Digit words from a result tile.
template <int NP>
__device__ __forceinline__ void tile_words(const float (&acc)[NP][8], uint32_t (&w)[NP][4]) {
#pragma unroll
  for (int h = 0; h < 4; ++h) {
    float a[NP], b[NP];
    tile_digits<NP>(acc, 2 * h, a);
    tile_digits<NP>(acc, 2 * h + 1, b);
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      const __half2 x = __floats2half2_rn(a[p], b[p]);
      w[p][h] = *reinterpret_cast<const uint32_t *>(&x);
    }
  }
}

// A block of planes for the left (A) or the right (B) side of a product.
template <int NP>
__device__ __forceinline__ void put_left(uint4 *blk, const uint32_t (&w)[NP][4]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int p = 0; p < NP; ++p) st_plane(blk + p * 32 + lane, make_uint4(w[p][0], w[p][1], w[p][2], w[p][3]));
}
template <int NP>
__device__ __forceinline__ void put_right(uint4 *blk, const uint32_t (&w)[NP][4]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int p = 0; p < NP; ++p) st_plane(blk + p * 32 + lane, make_uint4(w[p][0], w[p][2], w[p][1], w[p][3]));
}

__device__ __forceinline__ uint32_t transpose8(uint32_t v) {
  uint32_t r;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(v));
  return r;
}

// The first NP planes of a block's digit words as the transposed block.
template <int NP, int NW>
__device__ __forceinline__ void put_left_t(uint4 *blk, const uint32_t (&w)[NW][4]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int p = 0; p < NP; ++p)
    st_plane(blk + p * 32 + lane,
             make_uint4(transpose8(w[p][0]), transpose8(w[p][2]), transpose8(w[p][1]), transpose8(w[p][3])));
}
template <int NP, int NW>
__device__ __forceinline__ void put_right_t(uint4 *blk, const uint32_t (&w)[NW][4]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int p = 0; p < NP; ++p)
    st_plane(blk + p * 32 + lane,
             make_uint4(transpose8(w[p][0]), transpose8(w[p][1]), transpose8(w[p][2]), transpose8(w[p][3])));
}

// x 2^sh rounded to an integer (|result| < 2^62; 0 for a denormal x).
__device__ __forceinline__ long long fix(double x, int sh) {
  const long long b = __double_as_longlong(x);
  const int e = (int)((b >> 52) & 0x7ff);
  const long long m = e == 0 ? 0 : ((b & 0xfffffffffffffll) | 0x10000000000000ll);
  const int s = e - 1075 + sh;
  long long r;
  if (s >= 0) r = m << min(s, 10);
  else r = s < -60 ? 0 : (m + (1ll << (-s - 1))) >> -s;
  return b < 0 ? -r : r;
}

// t 2^e as a double, rounded to nearest; integer instructions only.
__device__ __forceinline__ double unfix(long long t, int e) {
  if (t == 0) return 0.0;
  unsigned long long u = (unsigned long long)(t < 0 ? -t : t);
  const int lz = __clzll((long long)u);
  u <<= lz;
  unsigned long long m = u >> 11;
  const unsigned rem = (unsigned)u & 0x7ffu;
  m += (rem > 0x400u || (rem == 0x400u && (m & 1))) ? 1 : 0;
  const long long b = (long long)(((unsigned long long)(63 - lz + e + 1022) << 52) + m);
  return __longlong_as_double(t < 0 ? (b | (long long)0x8000000000000000ull) : b);
}

// t 2^-56 in float32 (from the magnitude: a small negative t keeps its bits)
__device__ __forceinline__ float fix_to_float(long long t) {
  const unsigned long long u = (unsigned long long)(t < 0 ? -t : t);
  const float v = fmaf((float)(uint32_t)(u >> 32), 0x1p-24f, (float)(uint32_t)u * 0x1p-56f);
  return t < 0 ? -v : v;
}

// Smallest s with v <= 2^s (v > 0, finite).
__device__ __forceinline__ int exp_above(float v) {
  int e;
  const float m = frexpf(v, &e);
  return m == 0.5f ? e - 1 : e;
}

// Two maxima and two sums over the team, the same bits on every thread.
// sm: shared [32]; g: global [128] for a cluster. Ends with a team barrier.
struct Four {
  float m0, m1, s0, s1;
};
template <bool CL>
__device__ Four team_four(Team<CL> &tm, Four v, float4 *sm, float4 *g) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (int)(blockDim.x >> 5);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    v.m0 = fmaxf(v.m0, __shfl_xor_sync(0xffffffffu, v.m0, o));
    v.m1 = fmaxf(v.m1, __shfl_xor_sync(0xffffffffu, v.m1, o));
    v.s0 += __shfl_xor_sync(0xffffffffu, v.s0, o);
    v.s1 += __shfl_xor_sync(0xffffffffu, v.s1, o);
  }
  __syncthreads();  // the previous call's readers are done
  if (lane == 0) sm[wid] = make_float4(v.m0, v.m1, v.s0, v.s1);
  if constexpr (!CL) tm.sync(); else __syncthreads();
  Four r = {0.0f, 0.0f, 0.0f, 0.0f};
  auto add = [&](const float4 &x) {
    r.m0 = fmaxf(r.m0, x.x);
    r.m1 = fmaxf(r.m1, x.y);
    r.s0 += x.z;
    r.s1 += x.w;
  };
  for (int w = 0; w < nw; ++w) add(sm[w]);
  if constexpr (CL) {
    float4 *slot = g + 16 * (tm.phase & 1);
    ++tm.phase;
    if (threadIdx.x == 0) slot[tm.rank] = make_float4(r.m0, r.m1, r.s0, r.s1);
    tm.sync();
    r = {0.0f, 0.0f, 0.0f, 0.0f};
    for (int c = 0; c < tm.size; ++c) add(__ldcg(slot + c));
  }
  return r;
}
// fmaxf drops a NaN: sums carry it, so a caller that must see one looks there.

// 16-byte words of a lower tile's integrals: per lane 8 values (i, j) and
// their mirrors (j, i), 10 numbers of 8 bytes each
constexpr int kPairWords = 5 * 2 * 8 * 32;
constexpr int kOneWords = 8 * 32;  // S alone (without multipoles), pairs only
__host__ __device__ inline int pair_words(bool multipole) { return multipole ? kPairWords : kOneWords; }

// Workspace of this path (doubles), np = n rounded up to 16.
__host__ __device__ inline int64_t fast_size(int64_t n, int64_t nat, bool multipole) {
  const int64_t nb = blocks16(n), np2 = 256 * nb * nb;
  // planes of six digits are 12 bytes a value (3/2 doubles), of three 3/4;
  // the integrals S, D, Q in fixed point; potential and population tables
  return (5 * 3 * np2) / 2 + (2 * 3 * np2) / 4 + 2 * np2 + 6 * 16 * nb + 64 + 64 +
         nb * (nb + 1) / 2 * pair_words(multipole) * 2 + (n + 9 * nat) + 10 * n + 8;
}

// One copy per CTA in shared memory: as a local variable handed to functions
// its 300 bytes a thread filled the L1. Written by thread 0 between barriers.
struct Fast {
  int nb;
  uint4 *Xl, *XTl;           // X = L^-1 and its transpose
  uint4 *Fr, *Gl;            // F, F', weighted C^T (right); H, G, C^T (left)
  uint4 *Vl, *VT[2], *El;    // V (left), V^T (right), E^T (left, in G's memory)
  long long *Vm, *Vm2;       // vectors, weight 2^-kW, tile layout
  float *T, *R;              // tile layout (Vm2's memory)
  long long *td, *rd;        // diagonals of T and R
  double *lam;               // eigenvalue of each row of V
  int *xe, *xte, *inv;       // row exponents of X and X^T; row order
  float4 *red;
  long long *Ft;             // F and F' in fixed point, lower tiles (Vm2's memory)
  int4 *M;                   // S, D (3), Q (6) in fixed point, lower tiles: [5][pair, mirror][8][lane]
  long long *vo;             // orbital potential in fixed point
  int2 *vm;                  // atomic dipole and quadrupole potential, [9][nat]
  long long *pop;            // populations: charge and moments per orbital, [10][n]
  int eS, eD, eQ, eH;        // |S| <= 2^eS, ...
  int own_tables;            // vo and vm are in shared memory
  int nat, nm;               // atoms; 10 matrices in M, or 1 without multipoles
  int cur;                   // VT in use
  bool warm;                 // V holds vectors of an earlier problem
  float z0;                  // first rotation of the last problem
};

__device__ inline Fast fast_carve(double *base, int n, int nat, bool multipole) {
  Fast f;
  const int64_t nb = blocks16(n), np2 = 256 * nb * nb;
  f.nb = (int)nb;
  char *q = reinterpret_cast<char *>(base);
  q += (16 - ((uintptr_t)q & 15)) & 15;
  auto take = [&](int64_t bytes) {
    char *r = q;
    q += bytes;
    return r;
  };
  f.Xl = (uint4 *)take(12 * np2);
  f.XTl = (uint4 *)take(12 * np2);
  f.Fr = (uint4 *)take(12 * np2);
  f.Gl = (uint4 *)take(12 * np2);
  f.Vl = (uint4 *)take(12 * np2);
  f.VT[0] = (uint4 *)take(6 * np2);
  f.VT[1] = (uint4 *)take(6 * np2);
  f.El = f.Gl;
  f.Vm = (long long *)take(8 * np2);
  f.Vm2 = (long long *)take(8 * np2);
  f.T = (float *)f.Vm2;
  f.R = f.T + np2;
  f.red = (float4 *)take(32 * 16);
  f.td = (long long *)take(8 * 16 * nb);
  f.rd = (long long *)take(8 * 16 * nb);
  f.lam = (double *)take(8 * 16 * nb);
  f.xe = (int *)take(4 * 16 * nb);
  f.xte = (int *)take(4 * 16 * nb);
  f.inv = (int *)take(4 * 16 * nb);
  q += (16 - ((uintptr_t)q & 15)) & 15;
  f.Ft = f.Vm2;
  f.M = (int4 *)take(nb * (nb + 1) / 2 * pair_words(multipole) * 16);
  f.vo = (long long *)take(8 * (int64_t)n);
  f.vm = (int2 *)take(8 * 9 * (int64_t)nat);
  f.pop = (long long *)take(8 * 10 * (int64_t)n);
  f.own_tables = 0;
  f.nat = nat;
  f.nm = multipole ? 10 : 1;
  f.cur = 0;
  f.warm = false;
  f.z0 = 1.0f;
  return f;
}

// Warps of the team: this warp's index and their number. A CTA takes
// consecutive tiles, which share their A blocks in its L1.
template <bool CL>
__device__ __forceinline__ int team_warp(const Team<CL> &tm) {
  return tm.rank * (int)(blockDim.x >> 5) + (int)(threadIdx.x >> 5);
}
template <bool CL>
__device__ __forceinline__ int team_warps(const Team<CL> &tm) {
  return tm.size * (int)(blockDim.x >> 5);
}

// Tile t of the lower triangle (ti >= tj), row by row.
__device__ __forceinline__ void lower_tile(int t, int &ti, int &tj) {
  int r = (int)((sqrtf(8.0f * (float)t + 1.0f) - 1.0f) * 0.5f);
  while ((r + 1) * (r + 2) / 2 <= t) ++r;
  while (r * (r + 1) / 2 > t) --r;
  ti = r;
  tj = t - r * (r + 1) / 2;
}

// Row and column of value e of this lane in a tile.
__device__ __forceinline__ int tile_row(int e) { return ((threadIdx.x & 31) >> 2) + 8 * ((e >> 1) & 1); }
__device__ __forceinline__ int tile_col(int e) { return 8 * (e >> 2) + 2 * (threadIdx.x & 3) + (e & 1); }

// Digit planes of the row-major n x n matrix M (TR: of its transpose) whose
// row i is scaled by 2^-e[i], for the left side.
template <bool TR, bool CL>
__device__ __noinline__ void planes_of(Team<CL> &tm, int n, int nb, const double *M, uint4 *left,
                                       const int *ex) {
  for (int t = team_warp(tm); t < nb * nb; t += team_warps(tm)) {
    const int ti = t / nb, tj = t % nb;
    long long r[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int i = 16 * ti + tile_row(e), j = 16 * tj + tile_col(e);
      r[e] = 0;
      if (i < n && j < n) r[e] = fix(ld<CL>(TR ? M + (size_t)j * n + i : M + (size_t)i * n + j), kW - ldi<CL>(ex + i));
    }
    uint32_t w[kDig][4];
    cut_block<kDig>(r, w);
    put_left<kDig>(left + (size_t)t * kDig * 32, w);
  }
}

// |x| in float32, rounded up; infinity for |x| >= 2^127 and for a NaN. No
// FP64 instruction.
__device__ __forceinline__ float mag(double x) {
  const int hi = __double2hiint(x) & 0x7fffffff;
  if (hi >= 0x47e00000) return INFINITY;
  return hi < 0x38100000 ? 0.0f : __int_as_float(((hi - 0x38000000) << 3) + 8);
}

// Fixed point with kFix bits and a sign in two signed halves: h 2^29 + l,
// |h| <= 2^29, |l| <= 2^28. Five bits more than a float64 holds, since all
// entries of a matrix share one exponent.
constexpr int kFix = 58;
__device__ __forceinline__ int2 halves(long long m) {
  const int h = (int)((m + (1 << 28)) >> 29);
  return make_int2(h, (int)(m - ((long long)h << 29)));
}

// A product of two such numbers without its low x low part (at most 2^-60):
// three 32-bit multiply-adds in place of a float64 one, which costs nineteen
// times an IMAD's issue on this part. 20 products fit: |a0|, |a1| < 20 2^58.
__device__ __forceinline__ void mul_add(long long &a0, long long &a1, int2 x, int2 y) {
  a0 += (long long)x.x * y.x;
  a1 += (long long)x.x * y.y;
  a1 += (long long)x.y * y.x;
}

// S, D, Q in fixed point with their exponents (the factors of the Fock build
// and of the populations). False if an entry is not finite. Once per geometry.
template <bool CL>
__device__ __noinline__ bool fast_integrals(Team<CL> &tm, int n, Fast &f, const double *S, const double *H0,
                                            const double *D, const double *Q, int64_t mtot, float4 *sm) {
  const int64_t n2 = (int64_t)n * n;
  Four v = {0.0f, 0.0f, 0.0f, 0.0f};
  float h = 0.0f, s = 0.0f;
  for (int64_t t = tm.tid; t < n2; t += tm.nthr) {
    s = fmaxf(s, mag(S[t]));
    h = fmaxf(h, mag(H0[t]));
    if (f.nm > 1) {
      for (int c = 0; c < 3; ++c) v.m0 = fmaxf(v.m0, mag(D[c * mtot + t]));
      for (int c = 0; c < 6; ++c) v.m1 = fmaxf(v.m1, mag(Q[c * mtot + t]));
    }
  }
  const Four a = team_four(tm, v, sm, f.red), b = team_four(tm, Four{s, h, 0.0f, 0.0f}, sm, f.red);
  if (!(fmaxf(fmaxf(a.m0, a.m1), fmaxf(b.m0, b.m1)) < 0x1p60f)) return false;
  auto ex = [](float m) { return m > 0x1p-40f ? exp_above(m) : -40; };
  if (threadIdx.x == 0) {
    f.eS = ex(b.m0);
    f.eH = ex(b.m1);
    f.eD = ex(a.m0);
    f.eQ = ex(a.m1);
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, nlow = f.nb * (f.nb + 1) / 2;
  for (int t = team_warp(tm); t < nlow; t += team_warps(tm)) {
    int ti, tj;
    lower_tile(t, ti, tj);
    for (int e = 0; e < 8; ++e) {
      const int i = 16 * ti + tile_row(e), j = 16 * tj + tile_col(e);
      const bool in = i < n && j < n;
      for (int y = 0; y < (f.nm > 1 ? 2 : 1); ++y) {
        const int64_t o = y ? (int64_t)j * n + i : (int64_t)i * n + j;
        int2 m[10];
        m[0] = halves(in ? fix(S[o], kFix - f.eS) : 0);
        int4 *out = f.M + (size_t)t * pair_words(f.nm > 1) + (y * 8 + e) * 32 + lane;
        if (f.nm > 1) {
          for (int c = 0; c < 3; ++c) m[1 + c] = halves(in ? fix(D[c * mtot + o], kFix - f.eD) : 0);
          for (int c = 0; c < 6; ++c) m[4 + c] = halves(in ? fix(Q[c * mtot + o], kFix - f.eQ) : 0);
          for (int c = 0; c < 5; ++c) out[c * 512] = make_int4(m[2 * c].x, m[2 * c].y, m[2 * c + 1].x, m[2 * c + 1].y);
        } else {
          *out = make_int4(m[0].x, m[0].y, 0, 0);
        }
      }
    }
  }
  return true;
}

// Planes of X = L^-1 and of its transpose, rows scaled to a 2-norm in
// (1/2, 1]. False if a norm is not finite. Once per geometry.
template <bool CL>
__device__ __noinline__ bool fast_setup(Team<CL> &tm, int n, const double *X, Fast &f, float4 *sm) {
  const int lane = threadIdx.x & 31;
  float bad = 0.0f;
  for (int q = team_warp(tm); q < 2 * n; q += team_warps(tm)) {
    const int i = q >> 1;
    const bool tr = q & 1;
    float s = 0.0f;
    for (int k = lane; k < n; k += 32) {
      const float v = (float)ld<CL>(tr ? X + (size_t)k * n + i : X + (size_t)i * n + k);
      s = fmaf(v, v, s);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    const float nrm = sqrtf(s) * 1.000001f;
    const bool ok = nrm > 0x1p-60f && nrm < 0x1p60f;
    if (!ok) bad = 1.0f;
    const int ex = ok ? exp_above(nrm) : 0;
    if (lane == 0) (tr ? f.xte : f.xe)[i] = ex;
  }
  const Four r = team_four(tm, Four{bad, 0.0f, 0.0f, 0.0f}, sm, f.red);
  if (r.m0 > 0.0f) return false;
  planes_of<false>(tm, n, f.nb, X, f.Xl, f.xe);
  planes_of<true>(tm, n, f.nb, X, f.XTl, f.xte);
  tm.sync();
  return true;
}

// V = I (rows >= n zero).
template <bool CL>
__device__ __noinline__ void fast_identity(Team<CL> &tm, int n, Fast &f) {
  const int nb = f.nb, lane = threadIdx.x & 31;
  for (int t = team_warp(tm); t < nb * nb; t += team_warps(tm)) {
    const int ti = t / nb, tj = t % nb;
    long long v[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int i = 16 * ti + tile_row(e), j = 16 * tj + tile_col(e);
      v[e] = (i == j && i < n) ? 1ll << kW : 0;
      f.Vm[(((size_t)t * 4 + (e >> 1)) * 32 + lane) * 2 + (e & 1)] = v[e];
    }
    uint32_t w[kDig][4];
    cut_block<kDig>(v, w);
    put_left<kDig>(f.Vl + (size_t)t * kDig * 32, w);
    put_right_t<kDigLow>(f.VT[0] + ((size_t)tj * nb + ti) * kDigLow * 32, w);
  }
  if (threadIdx.x == 0) f.cur = 0;
  tm.sync();
}

// Lower tiles of a symmetric matrix in fixed point: value e of lane l of tile t.
__device__ __forceinline__ void put_tile(long long *F, int t, const long long (&v)[8]) {
  longlong2 *out = reinterpret_cast<longlong2 *>(F) + (size_t)t * 128 + (threadIdx.x & 31);
#pragma unroll
  for (int h = 0; h < 4; ++h) out[32 * h] = make_longlong2(v[2 * h], v[2 * h + 1]);
}
__device__ __forceinline__ void get_tile(const long long *F, int t, long long (&v)[8]) {
  const longlong2 *in = reinterpret_cast<const longlong2 *>(F) + (size_t)t * 128 + (threadIdx.x & 31);
#pragma unroll
  for (int h = 0; h < 4; ++h) {
    const longlong2 x = in[32 * h];
    v[2 * h] = x.x;
    v[2 * h + 1] = x.y;
  }
}

__device__ __forceinline__ long long shift(long long x, int left) {
  if (left >= 0) return x << min(left, 62);
  return left < -62 ? 0 : (x + (1ll << (-left - 1))) >> -left;
}

// The products of a step, a Fock build and a density: which tiles, what
// becomes of a result. One function per digit count: the instruction cache
// does not hold a copy of the tile loop for each product.
constexpr int kExpBias = 512;
enum Product : int {
  kStep,    // G = V F (planes), R = I - V V^T (float32, lower tiles)
  kProject, // T = G V^T (float32, lower tiles)
  kApply,   // V <- V + E^T V, planes of V and of its transpose
  kHalf,    // H = X F (planes), X lower triangular
  kFockX,    // F' = H X^T (fixed point, lower tiles)
  kCoeff,   // C^T = X^T V^T (planes), the mo lowest vectors
  kDensity, // P = C w C^T (fixed point, lower tiles); the diagonal's largest exponent + kExpBias
  kWeighted // the same in float64, both triangles
};

template <int NP, bool CL>
__device__ __noinline__ float tiles(Team<CL> &tm, int n, const Fast &f, Product what, int arg, int arg2, double *out) {
  const int nb = f.nb, nlow = nb * (nb + 1) / 2, lane = threadIdx.x & 31;
  const bool dens = what == kDensity || what == kWeighted;
  const int mb = what == kCoeff || dens ? (int)blocks16(arg) : nb;
  constexpr int S6 = kDig * 32, S3 = kDigLow * 32;
  const int row6 = nb * S6, row3 = nb * S3;
  const uint4 *VT = nullptr;
  uint4 *VN = nullptr;
  if (what == kApply) {  // only there: thread 0 turns f.cur right after it
    VT = f.VT[f.cur];
    VN = f.VT[f.cur ^ 1];
  }
  const int ntile = what == kStep                      ? nb * nb + nlow
                    : what == kApply || what == kHalf  ? nb * nb
                    : what == kCoeff                   ? nb * mb
                                                       : nlow;
  float sum = 0.0f;
  for (int t = team_warp(tm); t < ntile; t += team_warps(tm)) {
    int ti, tj, k0 = 0, k1 = nb, sa = S6, sb = S6;
    const uint4 *A, *B;
    bool left_b = false;   // B is stored for the left side
    bool square = false;  // a tile of the full matrix (else of the lower triangle)
    if (what == kApply || what == kHalf || (what == kStep && t < nb * nb)) {
      ti = t / nb;
      tj = t - ti * nb;
      square = true;
    } else if (what == kCoeff) {
      ti = t / mb;
      tj = t - ti * mb;
      square = true;
    } else {
      lower_tile(what == kStep ? t - nb * nb : t, ti, tj);
    }
    if (what == kHalf) {
      ti = nb - 1 - ti;  // the long rows first
      k1 = ti + 1;
    }
    if (what == kCoeff) k0 = ti;
    if (what == kFockX) k1 = tj + 1;
    if (dens) k1 = mb;
    if (what == kApply) {
      sa = sb = S3;
      A = f.El + (size_t)ti * row3;
      B = VT + (size_t)tj * row3;
    } else {
      A = (what == kStep ? f.Vl : what == kHalf ? f.Xl : what == kCoeff ? f.XTl : f.Gl) + (size_t)ti * row6;
      B = (what == kStep ? (square ? f.Fr : f.Vl)
           : what == kHalf || dens ? f.Fr
           : what == kFockX ? f.Xl : f.Vl) + (size_t)tj * row6;
      left_b = !(what == kHalf || dens || (what == kStep && square));
    }
    longlong2 vm[4];  // kApply: the vectors to update, loaded ahead
    if (NP == kDigLow && what == kApply) {
      const longlong2 *pv = reinterpret_cast<const longlong2 *>(f.Vm) + (size_t)(ti * nb + tj) * 128 + lane;
#pragma unroll
      for (int h = 0; h < 4; ++h) vm[h] = pv[32 * h];
    }
    float acc[NP][8];
    tile_nt<NP>(A, sa, B, sb, left_b, k0, k1, acc);
    const size_t blk = (size_t)ti * row6 + (size_t)tj * S6;
    if (NP == kDigLow && what == kApply) {
      longlong2 *pv = reinterpret_cast<longlong2 *>(f.Vm) + (size_t)(ti * nb + tj) * 128 + lane;
      long long c[8];
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        longlong2 v = vm[h];
        v.x += shift(tile_fix(acc, 2 * h), kW - kR - arg);  // weight 2^-kR 2^-ke to 2^-kW
        v.y += shift(tile_fix(acc, 2 * h + 1), kW - kR - arg);
        pv[32 * h] = v;
        c[2 * h] = v.x;
        c[2 * h + 1] = v.y;
      }
      uint4 *vt = VN + (size_t)tj * row3 + (size_t)ti * S3;
      if (arg2) {
        uint32_t w[kDig][4];
        cut_block<kDig>(c, w);
        put_left<kDig>(f.Vl + blk, w);
        put_right_t<kDigLow>(vt, w);
      } else {
        uint32_t w[kDigLow][4];
        cut_block<kDigLow>(c, w);
        put_left<kDigLow>(f.Vl + blk, w);
        put_right_t<kDigLow>(vt, w);
      }
    } else if (square) {
      uint32_t w[NP][4];
      tile_words<NP>(acc, w);
      put_left<NP>(f.Gl + blk, w);
    } else if (what == kStep || what == kProject) {
      const bool isr = what == kStep;
      const int tl = isr ? t - nb * nb : t;
      float4 *o = reinterpret_cast<float4 *>(isr ? f.R : f.T) + (size_t)tl * 64 + lane;
      float r[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const bool one = isr && ti == tj && tile_row(e) == tile_col(e) && 16 * ti + tile_row(e) < n;
        r[e] = tile_float(acc, e, one);
        if (isr) r[e] = -r[e];
      }
      o[0] = make_float4(r[0], r[1], r[2], r[3]);
      o[32] = make_float4(r[4], r[5], r[6], r[7]);
      if (ti == tj) {
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const int i = 16 * ti + tile_row(e);
          if (tile_row(e) == tile_col(e)) {
            const long long v = tile_fix(acc, e);
            if (isr) f.rd[i] = (i < n ? (1ll << kR) : 0) - v; else f.td[i] = v;
          }
        }
      }
    } else if (what == kFockX) {
      long long c[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        c[e] = tile_fix(acc, e);
        const int i = 16 * ti + tile_row(e), j = 16 * tj + tile_col(e);
        if (i < n && j < n) {
          const float y = ldexpf(tile_float(acc, e, false), f.xe[i] + f.xe[j]);
          sum = fmaf(ti == tj ? y : 2.0f * y, y, sum);
        }
      }
      put_tile(f.Ft, t, c);
    } else if (what == kDensity) {
      long long c[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        c[e] = tile_fix(acc, e);
        const int i = 16 * ti + tile_row(e);
        if (ti == tj && tile_row(e) == tile_col(e) && i < n && c[e] > 0)
          sum = fmaxf(sum, (float)(kExpBias + 2 * f.xte[i] + arg2 - kR + 64 - __clzll(c[e])));
      }
      put_tile(f.Ft, t, c);
    } else {
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const int i = 16 * ti + tile_row(e), j = 16 * tj + tile_col(e);
        if (i < n && j <= i) {
          const double v = unfix(tile_fix(acc, e), f.xte[i] + f.xte[j] + arg2 - kR);
          out[(size_t)i * n + j] = v;
          out[(size_t)j * n + i] = v;
        }
      }
    }
  }
  if (what != kFockX && what != kDensity) tm.sync();  // these two are followed by a team_four
  return sum;
}

// Rotations Z of the lower tiles over T, with the figures that scale them.
// lh, ll: shared, the eigenvalues as float32 pairs; lam: shared, in float64.
template <bool CL>
__device__ __noinline__ Four step_rotations(Team<CL> &tm, int n, const Fast &f, bool low, double *lam,
                                            float *lh, float *ll, float4 *sm) {
  const int nb = f.nb, nlow = nb * (nb + 1) / 2, lane = threadIdx.x & 31;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const double t = (double)(CL ? __ldcg(f.td + i) : f.td[i]) * 0x1p-58;
    const double r = (double)(CL ? __ldcg(f.rd + i) : f.rd[i]) * 0x1p-58;
    const double v = t * rcp_nr(1.0 - r);
    lam[i] = v;
    lh[i] = (float)v;
    ll[i] = (float)(v - (double)lh[i]);
  }
  __syncthreads();
  // inside a degenerate level couplings at the rounding level of T are left
  // alone (their ratio to the gap is noise); above the gap `far` every coupling
  // counts, since there thr / far is far below kFinal
  const float thr = low ? 0x1p-26f : 0x1p-54f, far = low ? 4.0f : 0x1p-22f;
  Four s = {0.0f, 0.0f, 0.0f, 0.0f};
  for (int t = team_warp(tm); t < nlow; t += team_warps(tm)) {
    int ti, tj;
    lower_tile(t, ti, tj);
    float4 *pt = reinterpret_cast<float4 *>(f.T) + (size_t)t * 64 + lane;
    const float4 *pr = reinterpret_cast<const float4 *>(f.R) + (size_t)t * 64 + lane;
    float z[8], r[8];
    *reinterpret_cast<float4 *>(z) = pt[0];
    *reinterpret_cast<float4 *>(z + 4) = pt[32];
    *reinterpret_cast<float4 *>(r) = pr[0];
    *reinterpret_cast<float4 *>(r + 4) = pr[32];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int i = 16 * ti + tile_row(e), j = 16 * tj + tile_col(e);
      float v = 0.0f;
      if (i < n && j < n) {
        if (i != j) {
          const float num = fmaf(0.5f * (lh[i] + lh[j]), r[e], z[e]);
          const float gap = (lh[j] - lh[i]) + (ll[j] - ll[i]);
          if (!(fabsf(num) < thr && fabsf(gap) < far)) {
            v = fabsf(num) < kZMax * fabsf(gap) ? __fdividef(num, gap)
                                                : (((__float_as_int(num) ^ __float_as_int(gap)) < 0) ? -kZMax : kZMax);
            if (!isfinite(num)) v = num;
          }
          if (i > j) {
            s.m0 = fmaxf(s.m0, fabsf(v));
            s.s0 = fmaf(v, v, s.s0);
          }
        }
        const float wgt = i > j ? 2.0f : (i == j ? 1.0f : 0.0f);
        s.m1 = fmaxf(s.m1, fabsf(r[e]));
        s.s1 = fmaf(wgt * r[e], r[e], s.s1);
      }
      z[e] = v;
    }
    pt[0] = *reinterpret_cast<float4 *>(z);
    pt[32] = *reinterpret_cast<float4 *>(z + 4);
  }
  return team_four(tm, s, sm, f.red);
}

// Planes of E^T, E = R / 2 + sc Z, scaled by 2^ke.
template <bool CL>
__device__ __noinline__ void step_update_planes(Team<CL> &tm, int n, const Fast &f, float sc, int ke) {
  const int nb = f.nb, nlow = nb * (nb + 1) / 2, lane = threadIdx.x & 31;
  const float up = ldexpf(1.0f, ke) * 0x1p30f;
  for (int t = team_warp(tm); t < nlow; t += team_warps(tm)) {
    int ti, tj;
    lower_tile(t, ti, tj);
    const float4 *pt = reinterpret_cast<const float4 *>(f.T) + (size_t)t * 64 + lane;
    const float4 *pr = reinterpret_cast<const float4 *>(f.R) + (size_t)t * 64 + lane;
    float z[8], r[8];
    *reinterpret_cast<float4 *>(z) = pt[0];
    *reinterpret_cast<float4 *>(z + 4) = pt[32];
    *reinterpret_cast<float4 *>(r) = pr[0];
    *reinterpret_cast<float4 *>(r + 4) = pr[32];
    int a[8], b[8];  // weight 2^-30; zero outside the matrix
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      a[e] = __float2int_rn(fmaf(-sc, z[e], 0.5f * r[e]) * up);  // E_ji
      b[e] = __float2int_rn(fmaf(sc, z[e], 0.5f * r[e]) * up);   // E_ij
    }
    uint32_t w[kDigLow][4];
    cut_words(a, w);
    put_left<kDigLow>(f.El + ((size_t)ti * nb + tj) * kDigLow * 32, w);
    if (ti != tj) {
      cut_words(b, w);
      put_left_t<kDigLow>(f.El + ((size_t)tj * nb + ti) * kDigLow * 32, w);
    }
  }
  tm.sync();
}

// Rows of V (and lam, shared) into ascending order of lam; sk: shared int64
// [n] scratch. Every CTA holds lam.
template <bool CL>
__device__ __noinline__ void fast_sort(Team<CL> &tm, int n, Fast &f, double *lam, double *sk, int *sflag) {
  const int nb = f.nb, lane = threadIdx.x & 31;
  long long *key = reinterpret_cast<long long *>(sk);
  if (threadIdx.x == 0) *sflag = 0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const long long b = __double_as_longlong(lam[i]);
    key[i] = b < 0 ? (b ^ 0x7fffffffffffffffll) : b;
  }
  __syncthreads();
  bool moved = false;
  for (int i = threadIdx.x + 1; i < n; i += blockDim.x) moved |= key[i - 1] > key[i];
  if (moved) *sflag = 1;
  __syncthreads();
  if (*sflag == 0) return;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const long long v = key[i];
    int r = 0;
    for (int j = 0; j < n; ++j) r += (key[j] < v) || (key[j] == v && j < i);
    if (tm.lead()) f.inv[r] = i;
    lam[r] = __longlong_as_double(v < 0 ? (v ^ 0x7fffffffffffffffll) : v);
  }
  tm.sync();
  for (int t = team_warp(tm); t < nb * nb; t += team_warps(tm)) {
    const int ti = t / nb, tj = t % nb;
    long long v[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int i = 16 * ti + tile_row(e);
      const int s = i < n ? ldi<CL>(f.inv + i) : i;
      // row s, same column: lane and value index of that row (pairs of values are one longlong2)
      const int sl = 4 * (s & 7) + (lane & 3), se = (e & 5) | (((s >> 3) & 1) << 1);
      v[e] = f.Vm[((((size_t)(s >> 4) * nb + tj) * 4 + (se >> 1)) * 32 + sl) * 2 + (se & 1)];
    }
    longlong2 *out = reinterpret_cast<longlong2 *>(f.Vm2) + (size_t)t * 128 + lane;
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      out[32 * h] = make_longlong2(v[2 * h], v[2 * h + 1]);
    }
    uint32_t w[kDig][4];
    cut_block<kDig>(v, w);
    put_left<kDig>(f.Vl + (size_t)t * kDig * 32, w);
    put_right_t<kDigLow>(f.VT[f.cur ^ 1] + ((size_t)tj * nb + ti) * kDigLow * 32, w);
  }
  tm.sync();
  if (threadIdx.x == 0) {
    f.cur ^= 1;
    long long *sw = f.Vm;
    f.Vm = f.Vm2;
    f.Vm2 = sw;
    f.Ft = sw;
    f.T = reinterpret_cast<float *>(f.Vm2);
    f.R = f.T + (size_t)256 * nb * nb;
  }
  __syncthreads();
}

// Eigenvectors (rows of V, ascending) and eigenvalues (lam, shared, every
// CTA; in units of 2^s) of the matrix whose planes, scaled by 2^-s to a
// Frobenius norm in (1/2, 1], are in f.Fr. False when they do not settle within
// max_steps. rotation: factor on the first bound of a step's rotations.
template <bool CL>
__device__ bool fast_eigen(Team<CL> &tm, int n, Fast &f, double *lam, double *sk, float *lh, float *ll, float4 *sm,
                           int max_steps, float rotation) {
  const bool warm = f.warm;
  const float z0 = f.z0;
  __syncthreads();
  if (threadIdx.x == 0) f.warm = false;
  if (!warm) fast_identity(tm, n, f);
  // the first rotation shrinks from one problem to the next as the SCF converges
  bool low = !warm || 0.5f * z0 > kZLow;
  float top = rotation * fmaxf(kZNorm, 0.2f * sqrtf((float)n)), zprev = 1.0f;
  bool stalled = false;
  for (int it = 0; it < max_steps; ++it) {
    if (low) {
      tiles<kDigLow>(tm, n, f, kStep, 0, 0, nullptr);
      tiles<kDigLow>(tm, n, f, kProject, 0, 0, nullptr);
    } else {
      tiles<kDig>(tm, n, f, kStep, 0, 0, nullptr);
      tiles<kDig>(tm, n, f, kProject, 0, 0, nullptr);
    }
    const Four s = step_rotations(tm, n, f, low, lam, lh, ll, sm);
    if (!isfinite(s.s0) || !(s.s1 < 1e4f)) {
      // too large a rotation: once more from the start with the bound that holds for any Z
      if (!(top > kZNorm)) return false;
      top = kZNorm;
      low = true;
      fast_identity(tm, n, f);
      continue;
    }
    // The singular values of I + E must stay below sqrt(3), where the R / 2
    // part contracts towards orthonormal rows. kZNorm bounds them for any Z by
    // its Frobenius norm; the many small rotations of a large problem have a
    // spectral norm far below that one (0.85 of 3.8 at n = 233), so the bound
    // grows with sqrt(n): 201 -> 143 coarse steps over an SCF at n = 233.
    const float zf = sqrtf(s.s0), rf = sqrtf(s.s1);
    const float lim = fmaxf(0.15f, top - 0.7f * rf);
    const float sc = zf > lim ? lim / zf : 1.0f;
    const float zm = s.m0 * sc;
    if (it == 0 && threadIdx.x == 0) f.z0 = zm;
    const bool last = !low && fmaxf(zf, rf) < kFinal;
    // scale of E for its digits: elements at most 1 and rows of norm at most 8,
    // which bounds every sum E^T V (up to n = 64 the one gives the other; above, by
    // the Frobenius norm)
    const float em = zm + 0.5f * s.m1, ef = n > 64 ? 1.4143f * sc * zf + 0.5f * rf : 0.0f;
    const int ke = min(em > 0x1p-50f ? -exp_above(em) : 50, 3 - exp_above(fmaxf(ef, 0x1p-60f)));
    step_update_planes(tm, n, f, sc, ke);
    // a coarse step that no longer shrinks the rotations has met its own rounding
    // (pairs closer than ~2^-20 of the norm): full steps from here on
    if (low && zm < 0x1p-6f && zm > 0.9f * zprev) stalled = true;
    zprev = zm;
    low = !last && !stalled && zm > kZLow;
    tiles<kDigLow>(tm, n, f, kApply, ke, low ? 0 : 1, nullptr);
    if (threadIdx.x == 0) f.cur ^= 1;  // read next after further barriers
    if (last) {
      __shared__ int sflag;
      fast_sort(tm, n, f, lam, sk, &sflag);
      if (threadIdx.x == 0) f.warm = true;
      return true;
    }
  }
  return false;
}

// Planes in f.Fr of the symmetric matrix in f.Ft, whose value (i, j) counts
// 2^(u(i) + u(j) + c) (ROWS: u the row exponents xe; else 0), scaled by 2^-s.
// The part below the diagonal is taken for both.
template <bool ROWS, bool CL>
__device__ __noinline__ void planes_of_tiles(Team<CL> &tm, int n, const Fast &f, int c) {
  const int nb = f.nb, nlow = nb * (nb + 1) / 2;
  for (int t = team_warp(tm); t < nlow; t += team_warps(tm)) {
    int ti, tj;
    lower_tile(t, ti, tj);
    long long v[8];
    get_tile(f.Ft, t, v);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int i = 16 * ti + tile_row(e), j = 16 * tj + tile_col(e);
      int k = c + kW;
      if constexpr (ROWS) {
        if (i < n && j < n) k += f.xe[i] + f.xe[j];
      }
      v[e] = (i < n && j <= i) ? shift(v[e], k) : 0;
    }
    uint32_t w[kDig][4];
    cut_block<kDig>(v, w);
    if (ti != tj) {
      put_right<kDig>(f.Fr + ((size_t)ti * nb + tj) * kDig * 32, w);
      put_right_t<kDig>(f.Fr + ((size_t)tj * nb + ti) * kDig * 32, w);
    } else {
#pragma unroll
      for (int e = 0; e < 8; ++e)
        if (tile_row(e) == tile_col(e)) v[e] = 0;
      uint32_t z[kDig][4];
      cut_block<kDig>(v, z);
#pragma unroll
      for (int p = 0; p < kDig; ++p) {
        const uint32_t y[4] = {transpose8(z[p][0]), transpose8(z[p][2]), transpose8(z[p][1]), transpose8(z[p][3])};
#pragma unroll
        for (int h = 0; h < 4; ++h) w[p][h] |= y[h];  // one of the two is zero
      }
      put_right<kDig>(f.Fr + ((size_t)ti * nb + ti) * kDig * 32, w);
    }
  }
  tm.sync();
}

// Exponent s of a scale 2^-s that puts a matrix of Frobenius norm sqrt(sum) to
// a norm in (1/2, 1].
__device__ __forceinline__ int norm_exp(float sum) {
  return sum > 0x1p-100f ? exp_above(sqrtf(sum) * 1.0001f) : 0;
}

// The Fock matrix F = H0 - S (v_i + v_j) / 2 - (T + T^T) / 2, T_ij = sum_c
// M_c,ij v_c(atom of j) (conversions.py:255-297), and F' = X F X^T, whose
// planes, scaled by 2^-s to a Frobenius norm in (1/2, 1], go to f.Fr. x: the
// potential (orbitals, atomic dipoles, quadrupoles); aoat: shared, atom of
// each orbital. All in fixed point: the float64 form (14 FMA a value) was
// bound by the FP64 pipe. False if a potential or norm is out of range.
template <bool CL>
__device__ __noinline__ bool fast_fock(Team<CL> &tm, int n, Fast &f, const double *H0, const double *x,
                                       const int *aoat, int &s, float4 *sm) {
  const int nb = f.nb, nlow = nb * (nb + 1) / 2, nat = f.nat;
  // exponents of the potentials, then their tables
  {
    float vo = 0.0f, vd = 0.0f, vq = 0.0f;
    const int N = f.nm > 1 ? n + 9 * nat : n;
    for (int t = threadIdx.x; t < N; t += blockDim.x) {
      const float m = mag(ld<CL>(x + t));
      if (t < n) vo = fmaxf(vo, m);
      else if (t < n + 3 * nat) vd = fmaxf(vd, m);
      else vq = fmaxf(vq, m);
    }
    // every CTA holds all values: the maxima need no exchange between them
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (int)(blockDim.x >> 5);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      vo = fmaxf(vo, __shfl_xor_sync(0xffffffffu, vo, o));
      vd = fmaxf(vd, __shfl_xor_sync(0xffffffffu, vd, o));
      vq = fmaxf(vq, __shfl_xor_sync(0xffffffffu, vq, o));
    }
    __syncthreads();
    if (lane == 0) sm[wid] = make_float4(vo, vd, vq, 0.0f);
    __syncthreads();
    for (int w = 0; w < nw; ++w) {
      vo = fmaxf(vo, sm[w].x);
      vd = fmaxf(vd, sm[w].y);
      vq = fmaxf(vq, sm[w].z);
    }
    if (!(fmaxf(vo, fmaxf(vd, vq)) < 0x1p60f)) return false;
    auto ex = [](float m) { return m > 0x1p-60f ? exp_above(m) : -60; };
    // one exponent E for all products: |M| 2^-eM and |v| 2^-(E - eM) are at most 1
    int E = max(f.eS + ex(vo) + 1, f.eH - 3);
    if (f.nm > 1) E = max(E, max(f.eD + ex(vd), f.eQ + ex(vq)));
    s = E;
    for (int t = tm.tid; t < f.nm * n; t += tm.nthr) f.pop[t] = 0;  // for this iteration's populations
    // tables in shared memory are every CTA's own
    for (int t = f.own_tables ? (int)threadIdx.x : tm.tid; t < N; t += f.own_tables ? (int)blockDim.x : tm.nthr) {
      const double v = ld<CL>(x + t);
      if (t < n) {
        f.vo[t] = fix(v, kFix - E + f.eS);
      } else if (t < n + 3 * nat) {
        const int u = t - n;
        f.vm[(u % 3) * nat + u / 3] = halves(fix(v, kFix - E + f.eD));
      } else {
        const int u = t - n - 3 * nat;
        f.vm[(3 + u % 6) * nat + u / 6] = halves(fix(v, kFix - E + f.eQ));
      }
    }
    tm.sync();
  }
  const int E = s;
  const uint64_t pol = stream_policy();
  Four sum = {0.0f, 0.0f, 0.0f, 0.0f};
  for (int t = team_warp(tm); t < nlow; t += team_warps(tm)) {
    int ti, tj;
    lower_tile(t, ti, tj);
    long long a0[8];
    int r[2], c[4];
#pragma unroll
    for (int k = 0; k < 2; ++k) r[k] = min(16 * ti + tile_row(2 * k), n - 1);
#pragma unroll
    for (int k = 0; k < 4; ++k) c[k] = min(16 * tj + tile_col((k >> 1) * 4 + (k & 1)), n - 1);
    if (f.nm > 1) {
      int ar[2], ac[4];
#pragma unroll
      for (int k = 0; k < 2; ++k) ar[k] = aoat[r[k]];
#pragma unroll
      for (int k = 0; k < 4; ++k) ac[k] = aoat[c[k]];
      // two matrices at a time (matrix 0 is S), first the pairs (i, j) with the
      // column atom's potential, then the mirrors (j, i) with the row atom's
      const int4 *M = f.M + (size_t)t * kPairWords + (threadIdx.x & 31);
      long long a1[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) a0[e] = a1[e] = 0;
#pragma unroll
      for (int m = 0; m < 5; ++m) {
        int4 x[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] = ld_stream(M + m * 512 + e * 32, pol);
        const int2 *u = f.vm + 2 * m * nat;
        int2 vc[4], uc[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          if (m) vc[k] = u[ac[k] - nat];
          uc[k] = u[ac[k]];
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const int kc = (e >> 2) * 2 + (e & 1);
          mul_add(a0[e], a1[e], make_int2(x[e].x, x[e].y),
                  m ? vc[kc] : halves(f.vo[r[(e >> 1) & 1]] + f.vo[c[kc]]));
          mul_add(a0[e], a1[e], make_int2(x[e].z, x[e].w), uc[kc]);
        }
      }
#pragma unroll
      for (int m = 0; m < 5; ++m) {
        int4 y[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) y[e] = ld_stream(M + m * 512 + 256 + e * 32, pol);
        const int2 *u = f.vm + 2 * m * nat;
        int2 vr[2], ur[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          if (m) vr[k] = u[ar[k] - nat];
          ur[k] = u[ar[k]];
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const int kr = (e >> 1) & 1;
          if (m) mul_add(a0[e], a1[e], make_int2(y[e].x, y[e].y), vr[kr]);
          mul_add(a0[e], a1[e], make_int2(y[e].z, y[e].w), ur[kr]);
        }
      }
      // in units of 2^(E - kFix)
#pragma unroll
      for (int e = 0; e < 8; ++e) a0[e] += a1[e] >> 29;
    } else {
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const int i = r[(e >> 1) & 1], j = c[(e >> 2) * 2 + (e & 1)];
        const int4 x = ld_stream(f.M + (size_t)t * kOneWords + e * 32 + (threadIdx.x & 31), pol);
        long long b0 = 0, b1 = 0;
        mul_add(b0, b1, make_int2(x.x, x.y), halves(f.vo[i] + f.vo[j]));
        a0[e] = b0 + (b1 >> 29);
      }
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int i = 16 * ti + tile_row(e), j = 16 * tj + tile_col(e);
      long long v = 0;
      if (i < n && j < n) v = fix(H0[(size_t)i * n + j], kFix - E) - ((a0[e] + 1) >> 1);
      a0[e] = v;
      const float y = fix_to_float(v);
      sum.s0 = fmaf(ti == tj ? y : 2.0f * y, y, sum.s0);
    }
    put_tile(f.Ft, t, a0);
  }
  const Four q = team_four(tm, sum, sm, f.red);
  const int sf = norm_exp(q.s0) + E - 2;  // fix_to_float took 2^-56 for 2^(E - kFix)
  planes_of_tiles<false>(tm, n, f, E - kFix - sf);
  tiles<kDig>(tm, n, f, kHalf, 0, 0, nullptr);
  sum.s0 = tiles<kDig>(tm, n, f, kFockX, 0, 0, nullptr);
  const Four p = team_four(tm, sum, sm, f.red);
  if (!(p.s0 < 0x1p100f)) return false;
  const int sn = norm_exp(p.s0);
  planes_of_tiles<true>(tm, n, f, -kR - sn);
  s = sn + sf;
  return true;
}

// Populations sum_k P_ki M_c,ki of every orbital i for the 10 (1) matrices,
// from the density in f.Ft (C w C^T with 0 <= w <= 2): f.pop[c n + i] in units
// of 2^(eP + eM - kFix + sh), sh returned. eP: every |P_ii| < 2^eP, hence
// every |P_ij|: one unit for all of P. (Units by the row norms of X, from which
// P is built, lose as many bits as these norms exceed P's entries, that is for
// an ill-conditioned S.) A lower tile serves the
// sums of its columns with the pairs and of its rows with their mirrors. Exact
// sums of fixed-point factors: the order of the atomics does not matter.
// In float64 (10 FMA a pair) this was bound by the FP64 pipe; here by the
// loads, 80 bytes a pair, which the tile order makes contiguous.
template <bool CL>
__device__ __noinline__ int fast_populations(Team<CL> &tm, int n, Fast &f, int eP) {
  const int lane = threadIdx.x & 31, nlow = f.nb * (f.nb + 1) / 2;
  int sh = 0;  // sums over n products of at most 2^58
  while ((16 << sh) < n) ++sh;
  const int nw = f.nm > 1 ? 5 : 1;
  const uint64_t pol = stream_policy();
  for (int t = team_warp(tm); t < nlow; t += team_warps(tm)) {
    int ti, tj;
    lower_tile(t, ti, tj);
    long long p[8];
    get_tile(f.Ft, t, p);
    int2 q[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int i = min(16 * ti + tile_row(e), n - 1), j = min(16 * tj + tile_col(e), n - 1);
      q[e] = halves(shift(p[e], f.xte[i] + f.xte[j] + 1 - kR + kFix - eP));
    }
    const int4 *M = f.M + (size_t)t * pair_words(f.nm > 1) + lane;
    const int mirror = f.nm > 1 ? 256 : 0;
    int4 x[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) x[e] = ld_stream(M + e * 32, pol);
#pragma unroll 1
    for (int m = 0; m < nw; ++m) {
#pragma unroll
      for (int half = 0; half < 2; ++half) {  // columns, then rows
        if (half == 1 && ti == tj) break;     // a diagonal tile holds every pair
        int4 xn[8];  // the next half's words, loaded ahead
        {
          const bool turn = half == 1 || ti == tj;
          const int4 *next = M + (turn ? (m + 1 < nw ? (m + 1) * 512 : 0) : m * 512 + mirror);
#pragma unroll
          for (int e = 0; e < 8; ++e) xn[e] = ld_stream(next + e * 32, pol);
        }
        long long s[4][2];
        {
          long long a0[4][2], a1[4][2];
#pragma unroll
          for (int k = 0; k < 4; ++k)
#pragma unroll
            for (int c = 0; c < 2; ++c) a0[k][c] = a1[k][c] = 0;
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            // columns: (e >> 2, e & 1); rows: (e >> 1) & 1
            const int k = half ? (e >> 1) & 1 : (e >> 2) * 2 + (e & 1);
            mul_add(a0[k][0], a1[k][0], q[e], make_int2(x[e].x, x[e].y));
            mul_add(a0[k][1], a1[k][1], q[e], make_int2(x[e].z, x[e].w));
          }
#pragma unroll
          for (int k = 0; k < 4; ++k)
#pragma unroll
            for (int c = 0; c < 2; ++c) s[k][c] = (a0[k][c] + (a1[k][c] >> 29) + ((1 << sh) >> 1)) >> sh;
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] = xn[e];
        // columns: over the 8 lanes of equal lane & 3; rows: over the 4 of equal lane >> 2
#pragma unroll
        for (int k = 0; k < (half ? 2 : 4); ++k)
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            long long v = s[k][c];
#pragma unroll
            for (int o = half ? 1 : 4; o < (half ? 4 : 32); o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            s[k][c] = v;
          }
        // lane l keeps one sum: column (k, c) from the lane >> 2 = 2 k + c of each
        // lane & 3; row (k, c) from the lane & 3 = 2 k + c of each lane >> 2
        const int w = half ? lane & 3 : lane >> 2;
        long long v = 0;
#pragma unroll
        for (int k = 0; k < (half ? 2 : 4); ++k)
#pragma unroll
          for (int c = 0; c < 2; ++c) v = w == 2 * k + c ? s[k][c] : v;
        const int k = w >> 1, c = 2 * m + (w & 1);
        const int o = half ? 16 * ti + (lane >> 2) + 8 * k : 16 * tj + 8 * (k >> 1) + 2 * (lane & 3) + (k & 1);
        if (o < n && c < f.nm)
          atomicAdd(reinterpret_cast<unsigned long long *>(f.pop + (size_t)c * n + o), (unsigned long long)v);
      }
    }
  }
  tm.sync();
  return sh;
}

// The density of f.Ft in float64 (both triangles).
template <bool CL>
__device__ __noinline__ void fast_store_density(Team<CL> &tm, int n, const Fast &f, double *out) {
  const int nlow = f.nb * (f.nb + 1) / 2;
  for (int t = team_warp(tm); t < nlow; t += team_warps(tm)) {
    int ti, tj;
    lower_tile(t, ti, tj);
    long long p[8];
    get_tile(f.Ft, t, p);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int i = 16 * ti + tile_row(e), j = 16 * tj + tile_col(e);
      if (i < n && j <= i) {
        const double v = unfix(p[e], f.xte[i] + f.xte[j] + 1 - kR);
        out[(size_t)i * n + j] = v;
        out[(size_t)j * n + i] = v;
      }
    }
  }
  tm.sync();
}

// One block of planes back as integers of weight 2^-kW.
__device__ __forceinline__ void join_block(const uint4 *blk, long long (&r)[8]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int e = 0; e < 8; ++e) r[e] = 0;
#pragma unroll
  for (int p = 0; p < kDig; ++p) {
    const uint4 w = blk[p * 32 + lane];
    const uint32_t u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      const __half2 x = *reinterpret_cast<const __half2 *>(&u[h]);
      r[2 * h] = r[2 * h] * 1024 + __half2int_rn(__low2half(x));
      r[2 * h + 1] = r[2 * h + 1] * 1024 + __half2int_rn(__high2half(x));
    }
  }
}

// C diag(w) C^T over the mo lowest orbitals from the planes of C^T in f.Gl;
// w(j): weight of orbital j, |w| <= 2^sw. To out (both triangles), or without
// it to f.Ft in units of 2^(xte_i + xte_j + sw - kR); the returned eP bounds
// this P, every |P_ii| < 2^eP.
template <bool CL, typename W>
__device__ __noinline__ int fast_density(Team<CL> &tm, int n, Fast &f, int mo, int sw, W w, double *out,
                                         float4 *sm) {
  const int nb = f.nb, mb = (int)blocks16(mo);
  for (int t = team_warp(tm); t < nb * mb; t += team_warps(tm)) {
    const int ti = t / mb, tj = t % mb;
    const size_t o = ((size_t)ti * nb + tj) * kDig * 32;
    long long r[8];
    join_block(f.Gl + o, r);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int j = 16 * tj + tile_col(e);
      const long long q = j < mo ? fix(w(j), 62 - sw) : 0;
      r[e] = __mul64hi(r[e] << 2, q);
    }
    uint32_t d[kDig][4];
    cut_block<kDig>(r, d);
    put_right<kDig>(f.Fr + o, d);
  }
  tm.sync();
  const float top = tiles<kDig>(tm, n, f, out != nullptr ? kWeighted : kDensity, mo, sw, out);
  if (out != nullptr) return 0;
  const Four r = team_four(tm, Four{top, 0.0f, 0.0f, 0.0f}, sm, f.red);
  return max((int)r.m0 - kExpBias, -60);
}

// The mo lowest orbitals' coefficients, row j of C (n x n, the rest zero).
template <bool CL>
__device__ __noinline__ void fast_orbitals(Team<CL> &tm, int n, const Fast &f, int mo, double *C) {
  const int nb = f.nb, mb = (int)blocks16(mo);
  for (int t = team_warp(tm); t < nb * mb; t += team_warps(tm)) {
    const int ti = t / mb, tj = t % mb;
    long long r[8];
    join_block(f.Gl + ((size_t)ti * nb + tj) * kDig * 32, r);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int i = 16 * ti + tile_row(e), j = 16 * tj + tile_col(e);
      if (i < n && j < mo) C[(size_t)j * n + i] = unfix(r[e], ldi<CL>(f.xte + i) - kW);
    }
  }
}

}  // namespace dxtb

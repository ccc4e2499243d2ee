// Symmetric eigenproblems and dense products of one molecule in 64-bit
// accuracy on the 16-bit tensor instructions, by a TEAM of CTAs (linalg.cuh).
//
// The FP64 pipe of this part issues 1.7 FMA per clock and SM, the 16-bit
// tensor instruction (mma.sync m16n8k16) 1020 (both measured): a product of
// 54-bit fixed-point operands cut into six digits of nine bits takes 21 digit
// products (those above 2^-54 of the largest), still ~28 times the FP64 rate,
// and is exact but for the digits left out: a digit product sum over 128
// terms stays below 2^24, where the float32 accumulator holds every integer.
// Sums over more terms are drained into 64-bit integers every 128.
//
// Fixed point: an operand's value is sum_p digit_p 2^(-9 (p + 1)) times a
// power of two kept beside the matrix (per matrix or per row); digits are
// balanced (|digit| <= 256) but the first, which takes the rest (|.| <= 2047,
// exact in fp16, so |value| < 4). Results are 64-bit integers of weight 2^-56.
//
// Digit planes are stored in the register layout of the instruction: a block
// of 16 x 16 values is one 16-byte word per lane and plane. The layout of the
// A operand (rows i, inner index k) with its four registers permuted is that
// of two B operands, so one set of planes serves on both sides of
// C = A B^T, and a result tile has the layout of an A operand.
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
// one molecule of 72 orbitals 36.9 -> 11.4 ms, of 233 orbitals (4 CTAs)
// 297 -> 82 ms, 256 molecules of 22-172 orbitals 225 -> 96 ms, with the same
// distance from the CPU oracle over the benchmark sets (|dE| <= 8e-12 Eh,
// |dF| <= 2.2e-11 Eh/Bohr).
#pragma once
#include <cuda_fp16.h>

#include "linalg.cuh"

namespace dxtb {

constexpr int kDig = 6;          // digits of a full operand
constexpr int kDigLow = 3;       // digits of the coarse steps and of the rotations
constexpr int kDrain = 8;        // k blocks of 16 per float32 accumulation
constexpr int kMaxSteps = 160;   // steps of one eigenproblem before it is given up
constexpr float kZMax = 0.4f;    // largest rotation of one pair in one step
constexpr float kZFinal = 0x1p-28f;  // a full step below this is the last (its error is quadratic)
constexpr float kZLow = 0x1p-10f;    // above this the next step is coarse

__host__ __device__ inline int64_t blocks16(int64_t n) { return (n + 15) / 16; }

__device__ __forceinline__ void mma16816(float *c, const uint4 &a, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3},{%4,%5,%6,%7},{%8,%9},{%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1));
}

// The 16 x 16 tile sum_k A[i][k] B[j][k] over the k blocks [k0, k1) with NP
// digits: A, B are the first blocks of the two block rows, PA, PB the planes
// stored per block. t[e], weight 2^-56: row g + 8 ((e >> 1) & 1), column
// 8 (e >> 2) + 2 q + (e & 1) for lane 4 g + q.
template <int NP, int PA, int PB>
__device__ __forceinline__ void tile_nt(const uint4 *A, const uint4 *B, int k0, int k1, long long (&t)[8]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int e = 0; e < 8; ++e) t[e] = 0;
  for (int kc = k0; kc < k1; kc += kDrain) {
    float acc[NP][8];
#pragma unroll
    for (int p = 0; p < NP; ++p)
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[p][e] = 0.0f;
    const int ke = min(kc + kDrain, k1);
    const uint4 *pa = A + (size_t)kc * PA * 32 + lane, *pb = B + (size_t)kc * PB * 32 + lane;
#pragma unroll 1
    for (int kb = kc; kb < ke; ++kb) {
      uint4 a[NP];
#pragma unroll
      for (int p = 0; p < NP; ++p) a[p] = pa[p * 32];
#pragma unroll
      for (int q = 0; q < NP; ++q) {
        const uint4 b = pb[q * 32];
#pragma unroll
        for (int p = 0; p < NP - q; ++p) {
          mma16816(acc[p + q], a[p], b.x, b.z);
          mma16816(acc[p + q] + 4, a[p], b.y, b.w);
        }
      }
      pa += PA * 32;
      pb += PB * 32;
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      // orders 0..2 have weights 2^-18, 2^-27, 2^-36, orders 3..5 2^-45 .. 2^-63
      const long long hi = (long long)__float2int_rn(acc[0][e]) * (1 << 18) +
                           (long long)__float2int_rn(acc[1][e]) * (1 << 9) + __float2int_rn(acc[2][e]);
      t[e] += hi * (1 << 20);
      if constexpr (NP > 3) {
        const long long lo = (long long)__float2int_rn(acc[3][e]) * (1 << 18) +
                             (long long)__float2int_rn(acc[4][e]) * (1 << 9) + __float2int_rn(acc[5][e]);
        t[e] += (lo + 64) >> 7;
      }
    }
  }
}

// Balanced digits of r (weight 2^-54), first digit first. With NP = 3 the
// value is rounded to 2^-27, which leaves the first three digits of NP = 6.
template <int NP>
__device__ __forceinline__ void cut(long long r, int (&d)[NP]) {
  const int hi = (int)((r + (1 << 26)) >> 27);
  if constexpr (NP == 6) {
    const int lo = (int)(r - ((long long)hi << 27));
    const int x1 = (lo + 256) >> 9, x2 = (x1 + 256) >> 9;
    d[5] = lo - (x1 << 9);
    d[4] = x1 - (x2 << 9);
    d[3] = x2;
  }
  const int y1 = (hi + 256) >> 9, y2 = (y1 + 256) >> 9;
  d[2] = hi - (y1 << 9);
  d[1] = y1 - (y2 << 9);
  d[0] = y2;
}

// Two digits as fp16. |d| <= 256: the bits of 1536 + d (unit spacing there)
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

template <int NP>
__device__ __forceinline__ void put_block(uint4 *blk, const uint32_t (&w)[NP][4]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int p = 0; p < NP; ++p) blk[p * 32 + lane] = make_uint4(w[p][0], w[p][1], w[p][2], w[p][3]);
}

__device__ __forceinline__ uint32_t transpose8(uint32_t v) {
  uint32_t r;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(v));
  return r;
}

// The first NP planes of a block's digit words as the transposed block.
template <int NP, int NW>
__device__ __forceinline__ void put_block_t(uint4 *blk, const uint32_t (&w)[NW][4]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int p = 0; p < NP; ++p)
    blk[p * 32 + lane] = make_uint4(transpose8(w[p][0]), transpose8(w[p][2]), transpose8(w[p][1]), transpose8(w[p][3]));
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

// Workspace of this path (doubles), np = n rounded up to 16.
__host__ __device__ inline int64_t fast_size(int64_t n) {
  const int64_t nb = blocks16(n), np2 = 256 * nb * nb;
  // planes of six digits are 12 bytes a value (3/2 doubles), of three 3/4
  return (5 * 3 * np2) / 2 + (3 * 3 * np2) / 4 + 2 * np2 + 6 * 16 * nb + 64 + 64;
}

struct Fast {
  int nb;
  uint4 *Xp, *XTp, *Fp, *Gp, *Vp, *VT[2], *Ep;
  long long *Vm, *Vm2;       // vectors, weight 2^-60, tile layout
  float *T, *R;              // tile layout (Vm2's memory)
  long long *td, *rd;        // diagonals of T and R
  double *lam;               // eigenvalue of each row of V
  int *xe, *xte, *inv;       // row exponents of X and X^T; row order
  float4 *red;
  int cur;                   // VT in use
  bool warm;                 // V holds vectors of an earlier problem
  float z0;                  // first rotation of the last problem
};

__device__ inline Fast fast_carve(double *base, int n) {
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
  f.Xp = (uint4 *)take(12 * np2);
  f.XTp = (uint4 *)take(12 * np2);
  f.Fp = (uint4 *)take(12 * np2);
  f.Gp = (uint4 *)take(12 * np2);
  f.Vp = (uint4 *)take(12 * np2);
  f.VT[0] = (uint4 *)take(6 * np2);
  f.VT[1] = (uint4 *)take(6 * np2);
  f.Ep = (uint4 *)take(6 * np2);
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
// row i is scaled by 2^-s(i).
template <bool TR, bool CL, typename S>
__device__ __noinline__ void planes_of(Team<CL> &tm, int n, int nb, const double *M, uint4 *out, S s) {
  for (int t = team_warp(tm); t < nb * nb; t += team_warps(tm)) {
    const int ti = t / nb, tj = t % nb;
    long long r[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int i = 16 * ti + tile_row(e), j = 16 * tj + tile_col(e);
      r[e] = 0;
      if (i < n && j < n) r[e] = fix(ld<CL>(TR ? M + (size_t)j * n + i : M + (size_t)i * n + j), 54 - s(i));
    }
    uint32_t w[kDig][4];
    cut_block<kDig>(r, w);
    put_block<kDig>(out + (size_t)t * kDig * 32, w);
  }
}

// Largest row sum of |M| (row-major, n x n) over the team; NaN or infinity
// gives a value that is not finite. Ends with a team barrier.
template <bool CL>
__device__ float team_inf_norm(Team<CL> &tm, int n, const double *M, float4 *sm, float4 *g) {
  const int lane = threadIdx.x & 31;
  float mx = 0.0f, all = 0.0f;
  for (int i = team_warp(tm); i < n; i += team_warps(tm)) {
    float s = 0.0f;
    for (int j = lane; j < n; j += 32) s += fabsf((float)ld<CL>(M + (size_t)i * n + j));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    mx = fmaxf(mx, s);
    all += s;
  }
  const Four f = team_four(tm, Four{mx, 0.0f, lane == 0 ? all : 0.0f, 0.0f}, sm, g);
  return isfinite(f.s0) ? f.m0 : f.s0;
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
    if (lane == 0) (tr ? f.xte : f.xe)[i] = ok ? exp_above(nrm) : 0;
  }
  const Four r = team_four(tm, Four{bad, 0.0f, 0.0f, 0.0f}, sm, f.red);
  if (r.m0 > 0.0f) return false;
  planes_of<false>(tm, n, f.nb, X, f.Xp, [&](int i) { return ldi<CL>(f.xe + i); });
  planes_of<true>(tm, n, f.nb, X, f.XTp, [&](int i) { return ldi<CL>(f.xte + i); });
  tm.sync();
  return true;
}

// V = I (rows >= n zero).
template <bool CL>
__device__ __noinline__ void fast_identity(Team<CL> &tm, int n, Fast &f) {
  const int nb = f.nb, lane = threadIdx.x & 31;
  for (int t = team_warp(tm); t < nb * nb; t += team_warps(tm)) {
    const int ti = t / nb, tj = t % nb;
    long long v[8], r[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int i = 16 * ti + tile_row(e), j = 16 * tj + tile_col(e);
      v[e] = (i == j && i < n) ? 1ll << 60 : 0;
      r[e] = v[e] >> 6;
      f.Vm[(((size_t)t * 4 + (e >> 1)) * 32 + lane) * 2 + (e & 1)] = v[e];
    }
    uint32_t w[kDig][4];
    cut_block<kDig>(r, w);
    put_block<kDig>(f.Vp + (size_t)t * kDig * 32, w);
    put_block_t<kDigLow>(f.VT[0] + ((size_t)tj * nb + ti) * kDigLow * 32, w);
  }
  f.cur = 0;
  tm.sync();
}

// One step's G = V F and R = I - V V^T (lower tiles).
template <int NP, bool CL>
__device__ __noinline__ void step_products(Team<CL> &tm, int n, const Fast &f) {
  const int nb = f.nb, nlow = nb * (nb + 1) / 2, lane = threadIdx.x & 31;
  for (int t = team_warp(tm); t < nb * nb + nlow; t += team_warps(tm)) {
    long long c[8];
    if (t < nb * nb) {
      const int ti = t / nb, tj = t % nb;
      tile_nt<NP, kDig, kDig>(f.Vp + (size_t)ti * nb * kDig * 32, f.Fp + (size_t)tj * nb * kDig * 32, 0, nb, c);
#pragma unroll
      for (int e = 0; e < 8; ++e) c[e] = (c[e] + 2) >> 2;
      uint32_t w[NP][4];
      cut_block<NP>(c, w);
      put_block<NP>(f.Gp + (size_t)t * kDig * 32, w);
    } else {
      int ti, tj;
      lower_tile(t - nb * nb, ti, tj);
      tile_nt<NP, kDig, kDig>(f.Vp + (size_t)ti * nb * kDig * 32, f.Vp + (size_t)tj * nb * kDig * 32, 0, nb, c);
      float4 *out = reinterpret_cast<float4 *>(f.R) + (size_t)(t - nb * nb) * 64 + lane;
      float r[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const int i = 16 * ti + tile_row(e), j = 16 * tj + tile_col(e);
        const long long v = (i == j && i < n) ? (1ll << 56) - c[e] : -c[e];
        r[e] = fix_to_float(v);
        if (i == j) f.rd[i] = v;
      }
      out[0] = make_float4(r[0], r[1], r[2], r[3]);
      out[32] = make_float4(r[4], r[5], r[6], r[7]);
    }
  }
  tm.sync();
}

// T = G V^T (lower tiles).
template <int NP, bool CL>
__device__ __noinline__ void step_project(Team<CL> &tm, const Fast &f) {
  const int nb = f.nb, nlow = nb * (nb + 1) / 2, lane = threadIdx.x & 31;
  for (int t = team_warp(tm); t < nlow; t += team_warps(tm)) {
    int ti, tj;
    lower_tile(t, ti, tj);
    long long c[8];
    tile_nt<NP, kDig, kDig>(f.Gp + (size_t)ti * nb * kDig * 32, f.Vp + (size_t)tj * nb * kDig * 32, 0, nb, c);
    float4 *out = reinterpret_cast<float4 *>(f.T) + (size_t)t * 64 + lane;
    float r[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      r[e] = fix_to_float(c[e]);
      if (ti == tj && tile_row(e) == tile_col(e)) f.td[16 * ti + tile_row(e)] = c[e];
    }
    out[0] = make_float4(r[0], r[1], r[2], r[3]);
    out[32] = make_float4(r[4], r[5], r[6], r[7]);
  }
  tm.sync();
}

// Rotations Z of the lower tiles over T, with the figures that scale them.
// lh, ll: shared, the eigenvalues as float32 pairs; lam: shared, in float64.
template <bool CL>
__device__ __noinline__ Four step_rotations(Team<CL> &tm, int n, const Fast &f, bool low, double *lam,
                                            float *lh, float *ll, float4 *sm) {
  const int nb = f.nb, nlow = nb * (nb + 1) / 2, lane = threadIdx.x & 31;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const double t = (double)(CL ? __ldcg(f.td + i) : f.td[i]) * 0x1p-56;
    const double r = (double)(CL ? __ldcg(f.rd + i) : f.rd[i]) * 0x1p-56;
    const double v = t * rcp_nr(1.0 - r);
    lam[i] = v;
    lh[i] = (float)v;
    ll[i] = (float)(v - (double)lh[i]);
  }
  __syncthreads();
  // couplings at the rounding level of T are left alone (inside a degenerate
  // level their ratio to the gap is noise)
  const float thr = low ? 0x1p-24f : 0x1p-51f;
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
          if (!(fabsf(num) < thr)) {
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
  const float up = ldexpf(1.0f, ke) * 0x1p27f;
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
    long long a[8], b[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int i = 16 * ti + tile_row(e), j = 16 * tj + tile_col(e);
      const bool in = i < n && j < n;
      a[e] = in ? (long long)__float2int_rn(fmaf(-sc, z[e], 0.5f * r[e]) * up) << 27 : 0;  // E_ji
      b[e] = in ? (long long)__float2int_rn(fmaf(sc, z[e], 0.5f * r[e]) * up) << 27 : 0;   // E_ij
    }
    uint32_t w[kDigLow][4];
    cut_block<kDigLow>(a, w);
    put_block<kDigLow>(f.Ep + ((size_t)ti * nb + tj) * kDigLow * 32, w);
    if (ti != tj) {
      cut_block<kDigLow>(b, w);
      put_block_t<kDigLow>(f.Ep + ((size_t)tj * nb + ti) * kDigLow * 32, w);
    }
  }
  tm.sync();
}

// V <- V + E^T V; NP planes of the new V (3 for a coarse next step) and the
// three of its transpose in the other buffer.
template <int NP, bool CL>
__device__ __noinline__ void step_apply(Team<CL> &tm, Fast &f, int ke) {
  const int nb = f.nb, lane = threadIdx.x & 31;
  const uint4 *VT = f.VT[f.cur];
  uint4 *VN = f.VT[f.cur ^ 1];
  for (int t = team_warp(tm); t < nb * nb; t += team_warps(tm)) {
    const int ti = t / nb, tj = t % nb;
    long long c[8];
    tile_nt<kDigLow, kDigLow, kDigLow>(f.Ep + (size_t)ti * nb * kDigLow * 32, VT + (size_t)tj * nb * kDigLow * 32, 0,
                                       nb, c);
    longlong2 *pv = reinterpret_cast<longlong2 *>(f.Vm) + (size_t)t * 128 + lane;
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      longlong2 v = pv[32 * h];
      const int sh = ke - 4;  // weight 2^-56 2^-ke to 2^-60
      auto move = [&](long long x) { return sh > 0 ? (x + (1ll << (sh - 1))) >> sh : x << -sh; };
      v.x += move(c[2 * h]);
      v.y += move(c[2 * h + 1]);
      pv[32 * h] = v;
      c[2 * h] = (v.x + 32) >> 6;
      c[2 * h + 1] = (v.y + 32) >> 6;
    }
    uint32_t w[NP][4];
    cut_block<NP>(c, w);
    put_block<NP>(f.Vp + (size_t)t * kDig * 32, w);
    put_block_t<kDigLow>(VN + ((size_t)tj * nb + ti) * kDigLow * 32, w);
  }
  f.cur ^= 1;
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
      v[2 * h] = (v[2 * h] + 32) >> 6;
      v[2 * h + 1] = (v[2 * h + 1] + 32) >> 6;
    }
    uint32_t w[kDig][4];
    cut_block<kDig>(v, w);
    put_block<kDig>(f.Vp + (size_t)t * kDig * 32, w);
    put_block_t<kDigLow>(f.VT[f.cur ^ 1] + ((size_t)tj * nb + ti) * kDigLow * 32, w);
  }
  f.cur ^= 1;
  long long *sw = f.Vm;
  f.Vm = f.Vm2;
  f.Vm2 = sw;
  f.T = reinterpret_cast<float *>(f.Vm2);
  f.R = f.T + (size_t)256 * nb * nb;
  tm.sync();
}

// Eigenvectors (rows of V, ascending) and eigenvalues (lam, shared, every
// CTA; in units of 2^s) of the matrix whose planes, scaled by 2^-s to a
// row-sum norm in (1, 2], are in f.Fp. False when the steps do not converge.
template <bool CL>
__device__ bool fast_eigen(Team<CL> &tm, int n, Fast &f, double *lam, double *sk, float *lh, float *ll, float4 *sm) {
  if (!f.warm) fast_identity(tm, n, f);
  // the first rotation shrinks from one problem to the next as the SCF converges
  bool low = !f.warm || 0.5f * f.z0 > kZLow;
  f.warm = false;
  for (int it = 0; it < kMaxSteps; ++it) {
    if (low) {
      step_products<kDigLow>(tm, n, f);
      step_project<kDigLow>(tm, f);
    } else {
      step_products<kDig>(tm, n, f);
      step_project<kDig>(tm, f);
    }
    const Four s = step_rotations(tm, n, f, low, lam, lh, ll, sm);
    if (!isfinite(s.s0) || !(s.s1 < 1e4f)) return false;
    // the singular values of I + E stay below sqrt(3), where the R / 2 part
    // contracts towards orthonormal rows
    const float zf = sqrtf(s.s0), rf = sqrtf(s.s1);
    const float lim = fmaxf(0.15f, 1.2f - 0.7f * rf);
    const float sc = zf > lim ? lim / zf : 1.0f;
    const float zm = s.m0 * sc;
    if (it == 0) f.z0 = zm;
    const bool last = !low && zm < kZFinal && s.m1 < 0x1p-26f;
    const float em = zm + 0.5f * s.m1;
    const int ke = em > 0x1p-50f ? -exp_above(em) : 50;
    step_update_planes(tm, n, f, sc, ke);
    low = !last && zm > kZLow;
    if (low) step_apply<kDigLow>(tm, f, ke); else step_apply<kDig>(tm, f, ke);
    if (last) {
      __shared__ int sflag;
      fast_sort(tm, n, f, lam, sk, &sflag);
      f.warm = true;
      return true;
    }
  }
  return false;
}

// F' = X F X^T into A (both triangles): F (row-major n x n) must be symmetric.
// Then the planes of F' in f.Fp scaled by 2^-s. False if a norm is not finite.
template <bool CL>
__device__ __noinline__ bool fast_transform(Team<CL> &tm, int n, Fast &f, const double *F, double *A, int &s,
                                            float4 *sm) {
  const int nb = f.nb;
  const float nf = team_inf_norm(tm, n, F, sm, f.red);
  if (!(nf < 0x1p60f)) return false;
  const int sf = nf > 0x1p-60f ? exp_above(nf * 1.0001f) - 1 : 0;
  planes_of<false>(tm, n, nb, F, f.Fp, [&](int) { return sf; });
  tm.sync();
  // H = X F: the planes of X are zero above the diagonal
  for (int t = team_warp(tm); t < nb * nb; t += team_warps(tm)) {
    const int ti = nb - 1 - t / nb, tj = t % nb;  // the long rows first
    long long c[8];
    tile_nt<kDig, kDig, kDig>(f.Xp + (size_t)ti * nb * kDig * 32, f.Fp + (size_t)tj * nb * kDig * 32, 0, ti + 1, c);
#pragma unroll
    for (int e = 0; e < 8; ++e) c[e] = (c[e] + 2) >> 2;
    uint32_t w[kDig][4];
    cut_block<kDig>(c, w);
    put_block<kDig>(f.Gp + ((size_t)ti * nb + tj) * kDig * 32, w);
  }
  tm.sync();
  for (int t = team_warp(tm); t < nb * (nb + 1) / 2; t += team_warps(tm)) {
    int ti, tj;
    lower_tile(t, ti, tj);
    long long c[8];
    tile_nt<kDig, kDig, kDig>(f.Gp + (size_t)ti * nb * kDig * 32, f.Xp + (size_t)tj * nb * kDig * 32, 0, tj + 1, c);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int i = 16 * ti + tile_row(e), j = 16 * tj + tile_col(e);
      if (i < n && j <= i) {
        const double v = unfix(c[e], ldi<CL>(f.xe + i) + ldi<CL>(f.xe + j) + sf - 56);
        A[(size_t)i * n + j] = v;
        A[(size_t)j * n + i] = v;
      }
    }
  }
  tm.sync();
  const float na = team_inf_norm(tm, n, A, sm, f.red);
  if (!(na < 0x1p60f)) return false;
  s = na > 0x1p-60f ? exp_above(na * 1.0001f) - 1 : 0;
  planes_of<false>(tm, n, nb, A, f.Fp, [&](int) { return s; });
  tm.sync();
  return true;
}

// Planes of C^T (rows: orbitals of the basis, columns: the mo lowest vectors)
// in f.Gp, rows scaled by 2^-xte.
template <bool CL>
__device__ __noinline__ void fast_coefficients(Team<CL> &tm, Fast &f, int mo) {
  const int nb = f.nb, mb = (int)blocks16(mo);
  for (int t = team_warp(tm); t < nb * mb; t += team_warps(tm)) {
    const int ti = t / mb, tj = t % mb;
    long long c[8];
    tile_nt<kDig, kDig, kDig>(f.XTp + (size_t)ti * nb * kDig * 32, f.Vp + (size_t)tj * nb * kDig * 32, ti, nb, c);
#pragma unroll
    for (int e = 0; e < 8; ++e) c[e] = (c[e] + 2) >> 2;
    uint32_t w[kDig][4];
    cut_block<kDig>(c, w);
    put_block<kDig>(f.Gp + ((size_t)ti * nb + tj) * kDig * 32, w);
  }
  tm.sync();
}

// One block of planes back as integers of weight 2^-54.
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
      r[2 * h] = r[2 * h] * 512 + __half2int_rn(__low2half(x));
      r[2 * h + 1] = r[2 * h + 1] * 512 + __half2int_rn(__high2half(x));
    }
  }
}

// out = C diag(w) C^T over the mo lowest orbitals (both triangles), from the
// planes of C^T in f.Gp; w(j): weight of orbital j, |w| <= 2^sw.
template <bool CL, typename W>
__device__ __noinline__ void fast_density(Team<CL> &tm, int n, Fast &f, int mo, int sw, W w, double *out) {
  const int nb = f.nb, mb = (int)blocks16(mo);
  for (int t = team_warp(tm); t < nb * mb; t += team_warps(tm)) {
    const int ti = t / mb, tj = t % mb;
    const size_t o = ((size_t)ti * nb + tj) * kDig * 32;
    long long r[8];
    join_block(f.Gp + o, r);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int j = 16 * tj + tile_col(e);
      const long long q = j < mo ? fix(w(j), 62 - sw) : 0;
      r[e] = __mul64hi(r[e] << 2, q);
    }
    uint32_t d[kDig][4];
    cut_block<kDig>(r, d);
    put_block<kDig>(f.Fp + o, d);
  }
  tm.sync();
  for (int t = team_warp(tm); t < nb * (nb + 1) / 2; t += team_warps(tm)) {
    int ti, tj;
    lower_tile(t, ti, tj);
    long long c[8];
    tile_nt<kDig, kDig, kDig>(f.Gp + (size_t)ti * nb * kDig * 32, f.Fp + (size_t)tj * nb * kDig * 32, 0, mb, c);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int i = 16 * ti + tile_row(e), j = 16 * tj + tile_col(e);
      if (i < n && j <= i) {
        const double v = unfix(c[e], ldi<CL>(f.xte + i) + ldi<CL>(f.xte + j) + sw - 56);
        out[(size_t)i * n + j] = v;
        out[(size_t)j * n + i] = v;
      }
    }
  }
  tm.sync();
}

// The mo lowest orbitals' coefficients, row j of C (n x n, the rest zero).
template <bool CL>
__device__ __noinline__ void fast_orbitals(Team<CL> &tm, int n, const Fast &f, int mo, double *C) {
  const int nb = f.nb, mb = (int)blocks16(mo);
  for (int t = team_warp(tm); t < nb * mb; t += team_warps(tm)) {
    const int ti = t / mb, tj = t % mb;
    long long r[8];
    join_block(f.Gp + ((size_t)ti * nb + tj) * kDig * 32, r);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int i = 16 * ti + tile_row(e), j = 16 * tj + tile_col(e);
      if (i < n && j < mo) C[(size_t)j * n + i] = unfix(r[e], ldi<CL>(f.xte + i) - 54);
    }
  }
}

}  // namespace dxtb

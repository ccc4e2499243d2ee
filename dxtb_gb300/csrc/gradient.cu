// Analytic nuclear gradient of the GFN1/GFN2-xTB energy at the converged SCF.
//
// The xTB free energy is variational in the density, so
//   dE/dR = dE/dR |_(P fixed) - sum_{mu nu} W_{mu nu} dS_{mu nu}/dR
// with the energy-weighted density W = C diag(f eps) C^T. The reference
// obtains the same quantity with autograd through the implicit SCF
// (calculators/types/autograd.py:84-196, scf/implicit/fixed_point.py:
// 250-431); GFN1's hand-written form is xtb/gfn1.py:185-408 and
// calculators/types/analytical.py:65-258.
//
// k_grad_pairs: one warp per shell pair with a d shell. Coefficient blocks for dS, dD, dQ
//   (from P, W, H0 scaling, orbital and multipole potentials) are
//   transformed back to the Cartesian basis, and the McMurchie-Davidson
//   tables with the bra shell raised/lowered give d/dA of every Cartesian
//   integral, contracted on the fly (no derivative integrals are stored).
//   The same warp adds the distance-polynomial term of H0 and the
//   coordination-number derivative of the self-energies.
// k_grad_terms: the s and p pairs, written out, and per atom ES2 (gamma), AES2
//   kernels and damping radii, repulsion.
// k_grad_cn: the chain rule through the coordination number.
#include "common.cuh"

namespace dxtb {

constexpr int gWarps = 4;
constexpr int gChunk = 16;   // primitive pairs staged per round
constexpr int kGradChunk = 4;  // shell pairs a warp looks through at a time
constexpr int gTab = 2 * 3 * 36;  // (T, dT) x axes x [a<=3][b<=2][e<=2] -> 216
constexpr int gNComp = 10;

__constant__ int g_cart[3][6][3] = {
    {{0, 0, 0}},
    {{0, 1, 0}, {0, 0, 1}, {1, 0, 0}},
    {{2, 0, 0}, {1, 1, 0}, {1, 0, 1}, {0, 2, 0}, {0, 1, 1}, {0, 0, 2}},
};
__constant__ int g_comp[gNComp][3] = {
    {0, 0, 0}, {1, 0, 0}, {0, 1, 0}, {0, 0, 1}, {2, 0, 0},
    {1, 1, 0}, {1, 0, 1}, {0, 2, 0}, {0, 1, 1}, {0, 0, 2},
};

__device__ __forceinline__ double gtrafo(int l, int m, int c) {
  if (l < 2) return m == c ? 1.0 : 0.0;
  const double s3 = 1.7320508075688772935274463415058723669;
  switch (m) {
    case 0: return c == 1 ? s3 : 0.0;
    case 1: return c == 4 ? s3 : 0.0;
    case 2: return c == 0 ? -0.5 : (c == 3 ? -0.5 : (c == 5 ? 1.0 : 0.0));
    case 3: return c == 2 ? s3 : 0.0;
    default: return c == 0 ? 0.5 * s3 : (c == 3 ? -0.5 * s3 : 0.0);
  }
}

// 1D Hermite tables T[a][b][e] for a <= la+1, b <= lb, e <= emax (about the
// ket centre), and the bra derivative dT[a][b][e] = 2 alpha T[a+1] - a T[a-1].
__device__ void md_tables_grad(int la, int lb, int emax, double alpha, double xpa, double xpb,
                               double x2p, double pref, double *T /*36*/, double *dT /*36*/) {
  double E[4][3][6];
  for (int a = 0; a < 4; ++a)
    for (int c = 0; c < 3; ++c)
      for (int t = 0; t < 6; ++t) E[a][c][t] = 0.0;
  E[0][0][0] = 1.0;
  const int la1 = la + 1;
  for (int a = 0; a < la1; ++a)
    for (int t = 0; t <= a + 1; ++t) {
      double v = xpa * E[a][0][t];
      if (t > 0) v += x2p * E[a][0][t - 1];
      if (t + 1 <= a) v += (t + 1) * E[a][0][t + 1];
      E[a + 1][0][t] = v;
    }
  for (int a = 0; a <= la1; ++a)
    for (int c = 0; c < lb; ++c)
      for (int t = 0; t <= a + c + 1; ++t) {
        double v = xpb * E[a][c][t];
        if (t > 0) v += x2p * E[a][c][t - 1];
        if (t + 1 <= a + c) v += (t + 1) * E[a][c][t + 1];
        E[a][c + 1][t] = v;
      }
  const double xpc = xpb;
  const double m10 = xpc, m20 = xpc * xpc + x2p, m21 = 2.0 * xpc;
  double Tl[4][3][3];
  for (int a = 0; a <= la1; ++a)
    for (int c = 0; c <= lb; ++c) {
      const double *e = E[a][c];
      Tl[a][c][0] = e[0];
      Tl[a][c][1] = emax >= 1 ? m10 * e[0] + e[1] : 0.0;
      Tl[a][c][2] = emax >= 2 ? m20 * e[0] + m21 * e[1] + 2.0 * e[2] : 0.0;
    }
  for (int a = 0; a <= la; ++a)
    for (int c = 0; c <= lb; ++c)
      for (int ee = 0; ee <= emax; ++ee) {
        const int o = (a * 3 + c) * 3 + ee;
        T[o] = pref * Tl[a][c][ee];
        double d = 2.0 * alpha * Tl[a + 1][c][ee];
        if (a > 0) d -= a * Tl[a - 1][c][ee];
        dT[o] = pref * d;
      }
}

struct GPair {
  int m, i, j, ti, tj, ai, aj, la, lb, na, nb;
  int64_t gi, gj, a0;
  double A[3], B[3];
};

// Powers that the parametrisations use, without pow(); uniform over a launch.
__device__ __forceinline__ double pow_p(double x, double p) {
  if (p == 3.0) return x * x * x;
  if (p == 4.0) return (x * x) * (x * x);
  if (p == 5.0) return (x * x) * (x * x) * x;
  if (p == 1.5) return x * sqrt(x);
  if (p == 1.0) return x;
  if (p == 0.5) return sqrt(x);
  return pow(x, p);
}

// Primitive pairs whose overlap is below e^-70 (4e-31) of the shells' norm are
// passed over: 2^-48 of a rounding error of the sum they would be added to.
constexpr double kNegligible = 70.0;

// Molecule and shells (i >= j) of pair k of the batch.
__device__ __forceinline__ void shell_pair(const dxtb_batch &b, int64_t k, int &m, int &i, int &j) {
  m = find_mol(b.pair_off, b.nmol, k);
  lower_pair(k - b.pair_off[m], i, j);
}

// One shell pair of the integral adjoint (one warp).
__device__ __forceinline__ void grad_pair(
    const dxtb_batch &b, const double *__restrict__ pf_, const int32_t *__restrict__ pi_tab,
    const double *__restrict__ cn, const double *__restrict__ P, const double *__restrict__ W,
    const double *__restrict__ S, const double *__restrict__ D, const double *__restrict__ vorb,
    const double *__restrict__ vdp, const double *__restrict__ vqp, int multipole,
    double *__restrict__ dedcn, double *__restrict__ grad, int64_t k, int lane, double *s_tab,
    double *s_esph, double *s_ecart) {

  GPair g;
  shell_pair(b, k, g.m, g.i, g.j);
  const int64_t s0 = b.shell_off[g.m];
  g.a0 = b.atom_off[g.m];
  g.gi = s0 + g.i;
  g.gj = s0 + g.j;
  g.ti = b.shell_type[g.gi];
  g.tj = b.shell_type[g.gj];
  g.ai = b.shell_atom[g.gi];
  g.aj = b.shell_atom[g.gj];
  for (int x = 0; x < 3; ++x) {
    g.A[x] = b.positions[3 * (g.a0 + g.ai) + x];
    g.B[x] = b.positions[3 * (g.a0 + g.aj) + x];
  }
  g.la = pi_(pi_tab, DXTB_I_L + g.ti);
  g.lb = pi_(pi_tab, DXTB_I_L + g.tj);
  g.na = pi_(pi_tab, DXTB_I_NPRIM + g.ti);
  g.nb = pi_(pi_tab, DXTB_I_NPRIM + g.tj);
  const int la = g.la, lb = g.lb, nsa = 2 * la + 1, nsb = 2 * lb + 1;
  const int64_t moff = b.mat_off[g.m], mtot = b.mat_off[b.nmol];
  const int n = (int)(b.ao_off[g.m + 1] - b.ao_off[g.m]);
  const int64_t o0 = b.ao_off[g.m];
  const int oi = b.shell_ao[g.gi], oj = b.shell_ao[g.gj];
  const bool same_atom = (g.ai == g.aj);
  const int zi = b.numbers[g.a0 + g.ai], zj = b.numbers[g.a0 + g.aj];

  // ---- H0 scaling of the pair (xtb/base.py:255-372) ----
  const double sei = pf(pf_, DXTB_P_LEVEL + g.ti) - pf(pf_, DXTB_P_KCN + g.ti) * cn[g.a0 + g.ai];
  const double sej = pf(pf_, DXTB_P_LEVEL + g.tj) - pf(pf_, DXTB_P_KCN + g.tj) * cn[g.a0 + g.aj];
  double fk = 1.0, pi = 1.0, dpi = 0.0, dist = 0.0;  // h = 0.5 (sei + sej) * pi * fk
  double d[3] = {g.B[0] - g.A[0], g.B[1] - g.A[1], g.B[2] - g.A[2]};
  if (!same_atom) {
    dist = sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2]);
    const double rsum = pf(pf_, DXTB_P_RAD + zi) + pf(pf_, DXTB_P_RAD + zj);
    const double rr = sqrt(dist / rsum);
    const double ki = pf(pf_, DXTB_P_SHPOLY + g.ti), kj = pf(pf_, DXTB_P_SHPOLY + g.tj);
    pi = (1.0 + ki * rr) * (1.0 + kj * rr);
    dpi = (ki * (1.0 + kj * rr) + kj * (1.0 + ki * rr)) * rr / (2.0 * dist);
    const int vi = pi_(pi_tab, DXTB_I_VALENCE + g.ti), vj = pi_(pi_tab, DXTB_I_VALENCE + g.tj);
    const double wexp = pf(pf_, DXTB_P_SCAL + DXTB_S_WEXP);
    const double zti = pf(pf_, DXTB_P_SLATER + g.ti), ztj = pf(pf_, DXTB_P_SLATER + g.tj);
    const double zfac = wexp == 0.0 ? 1.0 : pow_p(2.0 * sqrt(zti * ztj) / (zti + ztj), wexp);
    if (vi && vj) {
      const double den = pf(pf_, DXTB_P_EN + zi) - pf(pf_, DXTB_P_EN + zj);
      fk = pf(pf_, DXTB_P_KSHELL + la * 5 + lb) * zfac * pf(pf_, DXTB_P_KPAIR + zi * DXTB_MAXZ + zj) *
           (1.0 + pf(pf_, DXTB_P_SCAL + DXTB_S_ENSCALE) * den * den);
    } else {
      const double kpol = pf(pf_, DXTB_P_SCAL + DXTB_S_KPOL);
      const double kii = vi ? pf(pf_, DXTB_P_KSHELL + la * 6) : kpol;
      const double kjj = vj ? pf(pf_, DXTB_P_KSHELL + lb * 6) : kpol;
      fk = 0.5 * (kii + kjj) * zfac;
    }
  }
  const double h = 0.5 * (sei + sej) * pi * fk;

  // ---- coefficient blocks (spherical) ----
  double ps_part = 0.0, gconst[3] = {0.0, 0.0, 0.0};
  const int qa[6] = {0, 0, 1, 0, 1, 2}, qb[6] = {0, 1, 1, 2, 2, 2};
  const int q2comp[6] = {4, 5, 7, 6, 8, 9};  // (xx xy yy xz yz zz) -> component index
  const int64_t A0 = g.a0 + g.ai, B0 = g.a0 + g.aj;
  for (int o = lane; o < nsa * nsb; o += 32) {
    const int ma = o / nsb, mb = o % nsb;
    const int mu = oi + ma, nu = oj + mb;
    const int64_t e1 = moff + (int64_t)mu * n + nu;
    const double Pmn = P[e1], Smn = S[e1];
    ps_part += Pmn * Smn;
    double *es = s_esph + (size_t)o * gNComp;
    for (int c = 0; c < gNComp; ++c) es[c] = 0.0;
    if (same_atom) continue;
    const double cS2 = 2.0 * (Pmn * h - 0.5 * Pmn * (vorb[o0 + mu] + vorb[o0 + nu]) - W[e1]);
    if (!multipole) {
      es[0] = cS2;
      continue;
    }
    double cDA[3], cDB[3], cQA[6], cQB[6];
    for (int x = 0; x < 3; ++x) {
      cDB[x] = -Pmn * vdp[3 * B0 + x];
      cDA[x] = -Pmn * vdp[3 * A0 + x];
    }
    {
      double tA[6], tB[6];
      for (int c = 0; c < 6; ++c) {
        tB[c] = -Pmn * vqp[6 * B0 + c];
        tA[c] = -Pmn * vqp[6 * A0 + c];
      }
      const double trA = 0.5 * (tA[0] + tA[2] + tA[5]), trB = 0.5 * (tB[0] + tB[2] + tB[5]);
      for (int c = 0; c < 6; ++c) {
        const bool diag = (c == 0 || c == 2 || c == 5);
        cQA[c] = 1.5 * tA[c] - (diag ? trA : 0.0);
        cQB[c] = 1.5 * tB[c] - (diag ? trB : 0.0);
      }
    }
    double eS = cS2, eD[3];
    for (int x = 0; x < 3; ++x) {
      eS += cDA[x] * d[x];
      eD[x] = cDB[x] + cDA[x];
    }
    double DB[3];
    for (int x = 0; x < 3; ++x) DB[x] = D[x * mtot + e1];
    for (int c = 0; c < 6; ++c) {
      const int a = qa[c], bq = qb[c];
      eS += cQA[c] * d[a] * d[bq];
      eD[a] += cQA[c] * d[bq];
      eD[bq] += cQA[c] * d[a];
      es[q2comp[c]] = cQB[c] + cQA[c];
      // explicit dependence of the bra-centred moments on A
      gconst[bq] -= cQA[c] * (DB[a] + d[a] * Smn);
      gconst[a] -= cQA[c] * (DB[bq] + d[bq] * Smn);
    }
    for (int x = 0; x < 3; ++x) gconst[x] -= cDA[x] * Smn;
    es[0] = eS;
    for (int x = 0; x < 3; ++x) es[1 + x] = eD[x];
  }
  const double ps = warp_sum(ps_part);
  if (lane == 0) {
    // d E_h0 / d CN (self-energies): -kcn * sum_block P S * (pi * fk off-site)
    const double f = same_atom ? 1.0 : pi * fk;
    atomicAdd(&dedcn[A0], -pf(pf_, DXTB_P_KCN + g.ti) * f * ps);
    if (g.i != g.j) atomicAdd(&dedcn[B0], -pf(pf_, DXTB_P_KCN + g.tj) * f * ps);
  }
  if (same_atom) return;
  __syncwarp();

  // ---- back-transform coefficients to Cartesian: ec[a][b][comp] ----
  const int nca = (la + 1) * (la + 2) / 2, ncb = (lb + 1) * (lb + 2) / 2;
  const int ncomp = multipole ? gNComp : 1;
  const int emax = multipole ? 2 : 0;
  for (int o = lane; o < nca * ncb * ncomp; o += 32) {
    const int comp = o % ncomp, cb = (o / ncomp) % ncb, ca = o / (ncomp * ncb);
    double s = 0.0;
    for (int ma = 0; ma < nsa; ++ma) {
      const double ta = gtrafo(la, ma, ca);
      if (ta == 0.0) continue;
      for (int mb = 0; mb < nsb; ++mb) {
        const double tb = gtrafo(lb, mb, cb);
        if (tb == 0.0) continue;
        s += ta * tb * s_esph[(size_t)(ma * nsb + mb) * gNComp + comp];
      }
    }
    s_ecart[o] = s;
  }
  __syncwarp();

  // ---- contract with d/dA of the Cartesian integrals ----
  double gx = 0.0, gy = 0.0, gz = 0.0;
  const double r2 = dist * dist;
  const int npp = g.na * g.nb;
  const int nout = nca * ncb * ncomp;
  for (int c0 = 0; c0 < npp; c0 += gChunk) {
    const int cnt = min(gChunk, npp - c0);
    if (lane < cnt) {
      const int pp = c0 + lane;
      const int p1 = pp / g.nb, p2 = pp % g.nb;
      const double a = pf(pf_, DXTB_P_ALPHA + g.ti * DXTB_MAXPRIM + p1);
      const double bb = pf(pf_, DXTB_P_ALPHA + g.tj * DXTB_MAXPRIM + p2);
      const double ca = pf(pf_, DXTB_P_COEFF + g.ti * DXTB_MAXPRIM + p1);
      const double cb = pf(pf_, DXTB_P_COEFF + g.tj * DXTB_MAXPRIM + p2);
      const double oij = 1.0 / (a + bb), x2p = 0.5 * oij;
      const double sij = exp(-a * bb * oij * r2) * (kPi * sqrt(kPi)) * oij * sqrt(oij) * ca * cb;
      double *tab = s_tab + (size_t)lane * gTab;
      for (int x = 0; x < 3; ++x) {
        const double Pc = (a * g.A[x] + bb * g.B[x]) * oij;
        md_tables_grad(la, lb, emax, a, Pc - g.A[x], Pc - g.B[x], x2p, x == 0 ? sij : 1.0,
                       tab + 72 * x, tab + 72 * x + 36);
      }
    }
    __syncwarp();
    for (int o = lane; o < nout; o += 32) {
      const int comp = o % ncomp, cb = (o / ncomp) % ncb, ca = o / (ncomp * ncb);
      const double coef = s_ecart[o];
      if (coef == 0.0) continue;
      const int *na_ = g_cart[la][ca], *nb_ = g_cart[lb][cb], *ec = g_comp[comp];
      const int ix = (na_[0] * 3 + nb_[0]) * 3 + ec[0];
      const int iy = (na_[1] * 3 + nb_[1]) * 3 + ec[1];
      const int iz = (na_[2] * 3 + nb_[2]) * 3 + ec[2];
      double sx = 0.0, sy = 0.0, sz = 0.0;
      for (int q = 0; q < cnt; ++q) {
        const double *tab = s_tab + (size_t)q * gTab;
        const double Tx = tab[ix], dTx = tab[36 + ix];
        const double Ty = tab[72 + iy], dTy = tab[108 + iy];
        const double Tz = tab[144 + iz], dTz = tab[180 + iz];
        sx += dTx * Ty * Tz;
        sy += Tx * dTy * Tz;
        sz += Tx * Ty * dTz;
      }
      gx += coef * sx;
      gy += coef * sy;
      gz += coef * sz;
    }
    __syncwarp();
  }
  gx = warp_sum(gx + gconst[0]);
  gy = warp_sum(gy + gconst[1]);
  gz = warp_sum(gz + gconst[2]);
  if (lane == 0) {
    // distance polynomial of H0: 2 sum_block P h S * (dpi/dR) / pi along (A-B)/R
    const double dEdR = 2.0 * ps * h * dpi / pi;
    const double u[3] = {-d[0] / dist, -d[1] / dist, -d[2] / dist};  // (A - B) / R
    const double gv[3] = {gx + dEdR * u[0], gy + dEdR * u[1], gz + dEdR * u[2]};
    for (int x = 0; x < 3; ++x) {
      atomicAdd(&grad[3 * A0 + x], gv[x]);
      atomicAdd(&grad[3 * B0 + x], -gv[x]);
    }
  }
}

__global__ void __launch_bounds__(gWarps * 32)
    k_grad_pairs(dxtb_batch b, const double *__restrict__ pf_, const int32_t *__restrict__ pi_tab,
                 const double *__restrict__ cn, const double *__restrict__ P,
                 const double *__restrict__ W, const double *__restrict__ S,
                 const double *__restrict__ D, const double *__restrict__ vorb,
                 const double *__restrict__ vdp, const double *__restrict__ vqp, int multipole,
                 double *__restrict__ dedcn, double *__restrict__ grad, ClassFilter flt) {
  extern __shared__ double smem[];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double *s_tab = smem + (size_t)w * (gChunk * gTab + 2 * gNComp * 36);
  double *s_esph = s_tab + gChunk * gTab;      // [10][5][5] spherical coefficients
  double *s_ecart = s_esph + gNComp * 36;      // [6][6][10] Cartesian coefficients
  // kGradChunk pairs a warp at a time: each lane looks at one, then the warp takes
  // those with a d shell one after the other (they are neighbours: with 32 a
  // warp, sulfur-rich molecules left a tail of 0.3 ms)
  const int64_t npairs = b.pair_off[b.nmol];
  const int64_t step = (int64_t)gridDim.x * gWarps * kGradChunk;
  for (int64_t k0 = ((int64_t)blockIdx.x * gWarps + w) * kGradChunk; k0 < npairs; k0 += step) {
    bool mine = false;
    if (lane < kGradChunk && k0 + lane < npairs) {
      int m, i, j;
      shell_pair(b, k0 + lane, m, i, j);
      const int64_t s0 = b.shell_off[m];
      mine = in_class(flt, b, m) && (pi_(pi_tab, DXTB_I_L + b.shell_type[s0 + i]) > 1 ||
                                     pi_(pi_tab, DXTB_I_L + b.shell_type[s0 + j]) > 1);
    }
    for (unsigned todo = __ballot_sync(0xffffffffu, mine); todo != 0; todo &= todo - 1) {
      grad_pair(b, pf_, pi_tab, cn, P, W, S, D, vorb, vdp, vqp, multipole, dedcn, grad, k0 + __ffs(todo) - 1, lane,
                s_tab, s_esph, s_ecart);
      __syncwarp();  // the next pair reuses this warp's shared tables
    }
  }
}

// What the coefficients of a pair share (xtb/base.py:255-372).
struct GScale {
  double fk, pi, dpi, dist, h, d[3];
};
__device__ __forceinline__ GScale grad_scale(const dxtb_batch &b, const double *__restrict__ pf_,
                                             const int32_t *__restrict__ pi_tab, const double *__restrict__ cn,
                                             const GPair &g) {
  GScale q;
  const int zi = b.numbers[g.a0 + g.ai], zj = b.numbers[g.a0 + g.aj];
  const double sei = pf(pf_, DXTB_P_LEVEL + g.ti) - pf(pf_, DXTB_P_KCN + g.ti) * cn[g.a0 + g.ai];
  const double sej = pf(pf_, DXTB_P_LEVEL + g.tj) - pf(pf_, DXTB_P_KCN + g.tj) * cn[g.a0 + g.aj];
  q.fk = 1.0;
  q.pi = 1.0;
  q.dpi = 0.0;
  q.dist = 0.0;
#pragma unroll
  for (int x = 0; x < 3; ++x) q.d[x] = g.B[x] - g.A[x];
  if (g.ai != g.aj) {
    q.dist = sqrt(q.d[0] * q.d[0] + q.d[1] * q.d[1] + q.d[2] * q.d[2]);
    const double rsum = pf(pf_, DXTB_P_RAD + zi) + pf(pf_, DXTB_P_RAD + zj);
    const double rr = sqrt(q.dist / rsum);
    const double ki = pf(pf_, DXTB_P_SHPOLY + g.ti), kj = pf(pf_, DXTB_P_SHPOLY + g.tj);
    q.pi = (1.0 + ki * rr) * (1.0 + kj * rr);
    q.dpi = (ki * (1.0 + kj * rr) + kj * (1.0 + ki * rr)) * rr / (2.0 * q.dist);
    const int vi = pi_(pi_tab, DXTB_I_VALENCE + g.ti), vj = pi_(pi_tab, DXTB_I_VALENCE + g.tj);
    const double wexp = pf(pf_, DXTB_P_SCAL + DXTB_S_WEXP);
    const double zti = pf(pf_, DXTB_P_SLATER + g.ti), ztj = pf(pf_, DXTB_P_SLATER + g.tj);
    const double zfac = wexp == 0.0 ? 1.0 : pow_p(2.0 * sqrt(zti * ztj) / (zti + ztj), wexp);
    if (vi && vj) {
      const double den = pf(pf_, DXTB_P_EN + zi) - pf(pf_, DXTB_P_EN + zj);
      q.fk = pf(pf_, DXTB_P_KSHELL + g.la * 5 + g.lb) * zfac * pf(pf_, DXTB_P_KPAIR + zi * DXTB_MAXZ + zj) *
             (1.0 + pf(pf_, DXTB_P_SCAL + DXTB_S_ENSCALE) * den * den);
    } else {
      const double kpol = pf(pf_, DXTB_P_SCAL + DXTB_S_KPOL);
      const double kii = vi ? pf(pf_, DXTB_P_KSHELL + g.la * 6) : kpol;
      const double kjj = vj ? pf(pf_, DXTB_P_KSHELL + g.lb * 6) : kpol;
      q.fk = 0.5 * (kii + kjj) * zfac;
    }
  }
  q.h = 0.5 * (sei + sej) * q.pi * q.fk;
  return q;
}

// Coefficients of dS, dD, dQ (about B) for the matrix element (mu, nu) of an
// off-site pair, in the order of g_comp; gconst: the explicit dependence of the
// bra-centred moments on A.
template <int NC>
__device__ __forceinline__ void grad_coefs(const GPair &g, const GScale &q, double Pmn, double Smn, double vsum,
                                           double Wmn, const double *__restrict__ D, int64_t mtot, int64_t e1,
                                           const double *__restrict__ vdp, const double *__restrict__ vqp,
                                           double (&es)[NC], double (&gconst)[3]) {
  const double cS2 = 2.0 * (Pmn * q.h - 0.5 * Pmn * vsum - Wmn);
  es[0] = cS2;
  if constexpr (NC > 1) {
    const int qa[6] = {0, 0, 1, 0, 1, 2}, qb[6] = {0, 1, 1, 2, 2, 2};
    const int q2comp[6] = {4, 5, 7, 6, 8, 9};  // (xx xy yy xz yz zz) -> component index
    const int64_t A0 = g.a0 + g.ai, B0 = g.a0 + g.aj;
    double cDA[3], cDB[3], cQA[6], cQB[6], tA[6], tB[6], DB[3], eD[3];
#pragma unroll
    for (int x = 0; x < 3; ++x) {
      cDB[x] = -Pmn * vdp[3 * B0 + x];
      cDA[x] = -Pmn * vdp[3 * A0 + x];
      DB[x] = D[x * mtot + e1];
    }
#pragma unroll
    for (int c = 0; c < 6; ++c) {
      tB[c] = -Pmn * vqp[6 * B0 + c];
      tA[c] = -Pmn * vqp[6 * A0 + c];
    }
    const double trA = 0.5 * (tA[0] + tA[2] + tA[5]), trB = 0.5 * (tB[0] + tB[2] + tB[5]);
#pragma unroll
    for (int c = 0; c < 6; ++c) {
      const bool diag = (c == 0 || c == 2 || c == 5);
      cQA[c] = 1.5 * tA[c] - (diag ? trA : 0.0);
      cQB[c] = 1.5 * tB[c] - (diag ? trB : 0.0);
    }
    double eS = cS2;
#pragma unroll
    for (int x = 0; x < 3; ++x) {
      eS += cDA[x] * q.d[x];
      eD[x] = cDB[x] + cDA[x];
    }
#pragma unroll
    for (int c = 0; c < 6; ++c) {
      const int a = qa[c], bq = qb[c];
      eS += cQA[c] * q.d[a] * q.d[bq];
      eD[a] += cQA[c] * q.d[bq];
      eD[bq] += cQA[c] * q.d[a];
      es[q2comp[c]] = cQB[c] + cQA[c];
      gconst[bq] -= cQA[c] * (DB[a] + q.d[a] * Smn);
      gconst[a] -= cQA[c] * (DB[bq] + q.d[bq] * Smn);
    }
#pragma unroll
    for (int x = 0; x < 3; ++x) {
      gconst[x] -= cDA[x] * Smn;
      es[1 + x] = eD[x];
    }
    es[0] = eS;
  }
}

// One axis of a primitive pair: T[a][e] = the 1D integral with bra power a <= A,
// ket power C and moment e about the ket centre, dT = 2 alpha T[a + 1] - a T[a - 1],
// in units of the s-s overlap. The Hermite expansions E[a][c] written out.
template <int A, int C, int NC>
__device__ __forceinline__ void axis_table(double alpha, double xpa, double xpb, double x2p, double (&T)[A + 1][3],
                                           double (&dT)[A + 1][3]) {
  double E[3][3] = {{1.0, 0.0, 0.0}, {xpa, x2p, 0.0}, {0.0, 0.0, 0.0}};
  if constexpr (A > 0) {
    E[2][0] = fma(xpa, xpa, x2p);
    E[2][1] = 2.0 * xpa * x2p;
    E[2][2] = x2p * x2p;
  }
  if constexpr (C == 1) {
#pragma unroll
    for (int a = 0; a < A + 2; ++a) {
      const double e0 = E[a][0], e1 = E[a][1], e2 = E[a][2];
      E[a][0] = a > 0 ? fma(xpb, e0, e1) : xpb;
      E[a][1] = a > 0 ? fma(x2p, e0, a > 1 ? fma(xpb, e1, 2.0 * e2) : xpb * e1) : x2p;
      E[a][2] = a > 1 ? fma(xpb, e2, x2p * e1) : (a > 0 ? x2p * e1 : 0.0);
    }
  }
  const double m20 = fma(xpb, xpb, x2p), m21 = 2.0 * xpb;
  double R[3][3];
#pragma unroll
  for (int a = 0; a < A + 2; ++a) {
    R[a][0] = E[a][0];
    R[a][1] = NC > 1 ? fma(xpb, E[a][0], E[a][1]) : 0.0;
    R[a][2] = NC > 1 ? fma(m20, E[a][0], fma(m21, E[a][1], 2.0 * E[a][2])) : 0.0;
  }
#pragma unroll
  for (int e = 0; e < 3; ++e) {
    T[0][e] = R[0][e];
    dT[0][e] = 2.0 * alpha * R[1][e];
    if constexpr (A > 0) {
      T[1][e] = R[1][e];
      dT[1][e] = fma(2.0 * alpha, R[2][e], -R[0][e]);
    }
  }
}

// sum_comp c[comp] X Y Z with the derivative on each axis in turn; factors taken
// out axis by axis: 47 multiply-adds for 10 components instead of 90.
template <int NC>
__device__ __forceinline__ void grad_contract(const double *c, const double (&X)[3], const double (&dX)[3],
                                              const double (&Y)[3], const double (&dY)[3], const double (&Z)[3],
                                              const double (&dZ)[3], double &gx, double &gy, double &gz) {
  if constexpr (NC == 1) {
    const double yz = Y[0] * Z[0], cx = c[0] * X[0];
    gx = fma(c[0] * dX[0], yz, gx);
    gy = fma(cx, dY[0] * Z[0], gy);
    gz = fma(cx, Y[0] * dZ[0], gz);
  } else {
    // comps: 1, x, y, z, xx, xy, xz, yy, yz, zz
    auto row = [&](const double (&U)[3], double (&r)[6]) {
      r[0] = fma(c[4], U[2], fma(c[1], U[1], c[0] * U[0]));
      r[1] = fma(c[5], U[1], c[2] * U[0]);
      r[2] = c[7] * U[0];
      r[3] = fma(c[6], U[1], c[3] * U[0]);
      r[4] = c[8] * U[0];
      r[5] = c[9] * U[0];
    };
    auto cols = [&](const double (&r)[6], const double (&V)[3], double (&p)[3]) {
      p[0] = fma(r[2], V[2], fma(r[1], V[1], r[0] * V[0]));
      p[1] = fma(r[4], V[1], r[3] * V[0]);
      p[2] = r[5] * V[0];
    };
    double r[6], p[3];
    row(dX, r);
    cols(r, Y, p);
    gx = fma(p[2], Z[2], fma(p[1], Z[1], fma(p[0], Z[0], gx)));
    row(X, r);
    cols(r, dY, p);
    gy = fma(p[2], Z[2], fma(p[1], Z[1], fma(p[0], Z[0], gy)));
    cols(r, Y, p);
    gz = fma(p[2], dZ[2], fma(p[1], dZ[1], fma(p[0], dZ[0], gz)));
  }
}

// Primitive pair p of g: exponents, the s-s overlap (0: negligible) and the
// centre's distances.
struct GPrim {
  double a, x2p, sij, xpa[3], xpb[3];
};
__device__ __forceinline__ bool grad_prim(const double *__restrict__ pf_, const GPair &g, double r2, int p1, int p2,
                                          GPrim &q) {
  const double a = pf(pf_, DXTB_P_ALPHA + g.ti * DXTB_MAXPRIM + p1);
  const double bb = pf(pf_, DXTB_P_ALPHA + g.tj * DXTB_MAXPRIM + p2);
  const double oij = 1.0 / (a + bb), ex = a * bb * oij * r2;
  if (ex > kNegligible) return false;
  const double ca = pf(pf_, DXTB_P_COEFF + g.ti * DXTB_MAXPRIM + p1);
  const double cb = pf(pf_, DXTB_P_COEFF + g.tj * DXTB_MAXPRIM + p2);
  q.a = a;
  q.x2p = 0.5 * oij;
  q.sij = exp(-ex) * (kPi * sqrt(kPi)) * oij * sqrt(oij) * ca * cb;
#pragma unroll
  for (int x = 0; x < 3; ++x) {
    const double Pc = (a * g.A[x] + bb * g.B[x]) * oij;
    q.xpa[x] = Pc - g.A[x];
    q.xpb[x] = Pc - g.B[x];
  }
  return true;
}

// The pair's sums to the atoms: g = d/dA of its integrals, ps = sum P S.
__device__ __forceinline__ void grad_add(const GPair &g, const GScale &q, double ps, const double (&gr)[3],
                                         double *__restrict__ grad) {
  // distance polynomial of H0: 2 sum_block P h S * (dpi/dR) / pi along (A - B) / R
  const double dEdR = 2.0 * ps * q.h * q.dpi / (q.pi * q.dist);
  const int64_t A0 = g.a0 + g.ai, B0 = g.a0 + g.aj;
#pragma unroll
  for (int x = 0; x < 3; ++x) {
    const double v = gr[x] - dEdR * q.d[x];
    atomicAdd(&grad[3 * A0 + x], v);
    atomicAdd(&grad[3 * B0 + x], -v);
  }
}
__device__ __forceinline__ void grad_add_cn(const double *__restrict__ pf_, const GPair &g, const GScale &q, double ps,
                                            double *__restrict__ dedcn) {
  // d E_h0 / d CN (self-energies): -kcn * sum_block P S * (pi * fk off-site)
  const double f = q.pi * q.fk;
  atomicAdd(&dedcn[g.a0 + g.ai], -pf(pf_, DXTB_P_KCN + g.ti) * f * ps);
  if (g.i != g.j) atomicAdd(&dedcn[g.a0 + g.aj], -pf(pf_, DXTB_P_KCN + g.tj) * f * ps);
}

// One s-s or s-p shell pair of the integral adjoint on nsub lanes, of which this
// is lane `part` (its primitive pairs; part 0 also the constant terms), the s shell
// on the bra (a p-s pair is evaluated as its s-p mirror, which holds the same
// two matrix elements; the pair's contribution is symmetric under exchanging
// bra and ket); the spherical transform is the identity.
template <int LB, int NC>
__device__ __forceinline__ void grad_pair_sp(
    const dxtb_batch &b, const double *__restrict__ pf_, const int32_t *__restrict__ pi_tab,
    const double *__restrict__ cn, const double *__restrict__ P, const double *__restrict__ W,
    const double *__restrict__ S, const double *__restrict__ D, const double *__restrict__ vorb,
    const double *__restrict__ vdp, const double *__restrict__ vqp, const GPair &g, int part, int nsub, GScale &q,
    double &ps, double (&gr)[3]) {
  constexpr int NSB = 2 * LB + 1;
  const int64_t moff = b.mat_off[g.m], mtot = b.mat_off[b.nmol], o0 = b.ao_off[g.m];
  const int n = (int)(b.ao_off[g.m + 1] - o0);
  const int oi = b.shell_ao[g.gi], oj = b.shell_ao[g.gj];
  const bool same_atom = (g.ai == g.aj);
  q = grad_scale(b, pf_, pi_tab, cn, g);
  double gconst[3] = {0.0, 0.0, 0.0};
  double es[NSB][NC];
#pragma unroll
  for (int mb = 0; mb < NSB; ++mb) {
    const int mu = oi, nu = oj + mb;
    const int64_t e1 = moff + (int64_t)mu * n + nu;
    const double Pmn = P[e1], Smn = S[e1];
    ps += Pmn * Smn;
    if (!same_atom)
      grad_coefs<NC>(g, q, Pmn, Smn, vorb[o0 + mu] + vorb[o0 + nu], W[e1], D, mtot, e1, vdp, vqp, es[mb], gconst);
  }
  if (same_atom) return;
  if (part == 0) {
#pragma unroll
    for (int x = 0; x < 3; ++x) gr[x] = gconst[x];
  }
  // contraction with d/dA of the Cartesian integrals (moments about B)
  const double r2 = q.dist * q.dist;
  for (int p = part; p < g.na * g.nb; p += nsub) {
    GPrim w;
    if (!grad_prim(pf_, g, r2, p / g.nb, p % g.nb, w)) continue;
    double T[3][2][3], dT[3][2][3];  // [axis][ket power]
#pragma unroll
    for (int x = 0; x < 3; ++x) {
      axis_table<0, 0, NC>(w.a, w.xpa[x], w.xpb[x], w.x2p, reinterpret_cast<double (&)[1][3]>(T[x][0]),
                           reinterpret_cast<double (&)[1][3]>(dT[x][0]));
      if constexpr (LB == 1)
        axis_table<0, 1, NC>(w.a, w.xpa[x], w.xpb[x], w.x2p, reinterpret_cast<double (&)[1][3]>(T[x][1]),
                             reinterpret_cast<double (&)[1][3]>(dT[x][1]));
    }
    double s[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int cb = 0; cb < NSB; ++cb) {
      // p order (y, z, x): component cb raises axis (cb + 1) % 3
      const int px = LB == 1 && cb == 2, py = LB == 1 && cb == 0, pz = LB == 1 && cb == 1;
      grad_contract<NC>(es[cb], T[0][px], dT[0][px], T[1][py], dT[1][py], T[2][pz], dT[2][pz], s[0], s[1], s[2]);
    }
#pragma unroll
    for (int x = 0; x < 3; ++x) gr[x] = fma(w.sij, s[x], gr[x]);
  }
}

// One p-p pair on 16 lanes: a lane per matrix element for the coefficients
// (es: shared, [9][NC]), then a lane per primitive pair.
template <int NC>
__device__ __forceinline__ void grad_pair_pp(
    const dxtb_batch &b, const double *__restrict__ pf_, const int32_t *__restrict__ pi_tab,
    const double *__restrict__ cn, const double *__restrict__ P, const double *__restrict__ W,
    const double *__restrict__ S, const double *__restrict__ D, const double *__restrict__ vorb,
    const double *__restrict__ vdp, const double *__restrict__ vqp, double *__restrict__ dedcn,
    double *__restrict__ grad, const GPair &g, bool active, double *es) {
  const int hl = threadIdx.x & 15;
  const bool same_atom = (g.ai == g.aj);
  double ps = 0.0, gr[3] = {0.0, 0.0, 0.0};
  GScale q = {};
  if (active) {
    const int64_t moff = b.mat_off[g.m], mtot = b.mat_off[b.nmol], o0 = b.ao_off[g.m];
    const int n = (int)(b.ao_off[g.m + 1] - o0);
    q = grad_scale(b, pf_, pi_tab, cn, g);
    if (hl < 9) {
      const int mu = b.shell_ao[g.gi] + hl / 3, nu = b.shell_ao[g.gj] + hl % 3;
      const int64_t e1 = moff + (int64_t)mu * n + nu;
      const double Pmn = P[e1], Smn = S[e1];
      ps = Pmn * Smn;
      if (!same_atom) {
        double c[NC];
        grad_coefs<NC>(g, q, Pmn, Smn, vorb[o0 + mu] + vorb[o0 + nu], W[e1], D, mtot, e1, vdp, vqp, c, gr);
#pragma unroll
        for (int k = 0; k < NC; ++k) es[hl * NC + k] = c[k];
      }
    }
  }
  __syncwarp();
  if (active && !same_atom) {
    const double r2 = q.dist * q.dist;
    for (int p = hl; p < g.na * g.nb; p += 16) {
      GPrim w;
      if (!grad_prim(pf_, g, r2, p / g.nb, p % g.nb, w)) continue;
      double s[3] = {0.0, 0.0, 0.0};
#pragma unroll
      for (int cb = 0; cb < 3; ++cb) {
        double T[3][2][3], dT[3][2][3];  // [axis][bra power], the ket's power on axis (cb + 1) % 3
#pragma unroll
        for (int x = 0; x < 3; ++x) {
          if (x == (cb + 1) % 3) axis_table<1, 1, NC>(w.a, w.xpa[x], w.xpb[x], w.x2p, T[x], dT[x]);
          else axis_table<1, 0, NC>(w.a, w.xpa[x], w.xpb[x], w.x2p, T[x], dT[x]);
        }
#pragma unroll
        for (int ca = 0; ca < 3; ++ca) {
          const int px = ca == 2, py = ca == 0, pz = ca == 1;
          grad_contract<NC>(es + (ca * 3 + cb) * NC, T[0][px], dT[0][px], T[1][py], dT[1][py], T[2][pz], dT[2][pz],
                            s[0], s[1], s[2]);
        }
      }
#pragma unroll
      for (int x = 0; x < 3; ++x) gr[x] = fma(w.sij, s[x], gr[x]);
    }
  }
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) {
    ps += __shfl_xor_sync(0xffffffffu, ps, o);
#pragma unroll
    for (int x = 0; x < 3; ++x) gr[x] += __shfl_xor_sync(0xffffffffu, gr[x], o);
  }
  if (active && hl == 0) {
    grad_add_cn(pf_, g, q, ps, dedcn);
    if (!same_atom) grad_add(g, q, ps, gr, grad);
  }
}

__device__ __forceinline__ void grad_pair_setup(const dxtb_batch &b, const int32_t *__restrict__ pi_tab, GPair &g) {
  const int64_t s0 = b.shell_off[g.m];
  g.a0 = b.atom_off[g.m];
  g.gi = s0 + g.i;
  g.gj = s0 + g.j;
  g.ti = b.shell_type[g.gi];
  g.tj = b.shell_type[g.gj];
  g.la = pi_(pi_tab, DXTB_I_L + g.ti);
  g.lb = pi_(pi_tab, DXTB_I_L + g.tj);
  g.ai = b.shell_atom[g.gi];
  g.aj = b.shell_atom[g.gj];
#pragma unroll
  for (int x = 0; x < 3; ++x) {
    g.A[x] = b.positions[3 * (g.a0 + g.ai) + x];
    g.B[x] = b.positions[3 * (g.a0 + g.aj) + x];
  }
  g.na = pi_(pi_tab, DXTB_I_NPRIM + g.ti);
  g.nb = pi_(pi_tab, DXTB_I_NPRIM + g.tj);
}

__device__ __forceinline__ double exp_count_d(double r, double r0, double k, double *dc) {
  const double c = 1.0 / (1.0 + exp(-k * (r0 / r - 1.0)));
  *dc = -c * (1.0 - c) * k * r0 / (r * r);
  return c;
}

constexpr int kGradAtoms = 8;  // atoms a CTA takes

// ES2, AES2 and repulsion of kGradAtoms atoms of molecule m with all others, a
// warp per atom and a lane per partner. (A thread per atom was a serial chain
// of up to 60 pairs with four pow() each: 2.6 ms a size class.) sm: 2 nsh
// doubles, nat + 1 ints.
__device__ __forceinline__ void grad_atoms(const dxtb_batch &b, const double *__restrict__ pf_,
                                           const int32_t *__restrict__ pi_tab, const double *__restrict__ cn,
                                           const double *__restrict__ mrad, const double *__restrict__ q,
                                           const double *__restrict__ dp, const double *__restrict__ qp,
                                           int multipole, double *__restrict__ dedcn, double *__restrict__ grad,
                                           int m, int first, double *sm) {
  const int64_t a0 = b.atom_off[m], s0 = b.shell_off[m], o0 = b.ao_off[m];
  const int nat = (int)(b.atom_off[m + 1] - a0), nsh = (int)(b.shell_off[m + 1] - s0);
  if (first >= nat) return;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int avg_kind = pi_(pi_tab, DXTB_I_SCAL + DXTB_IS_AVERAGE);
  double *qsh = sm, *hard = sm + nsh;                // charge; hardness, for the harmonic mean its inverse
  int *sfirst = reinterpret_cast<int *>(hard + nsh); // [nat + 1] first shell of each atom
  for (int s = threadIdx.x; s < nsh; s += blockDim.x) {
    const int t = b.shell_type[s0 + s], at = b.shell_atom[s0 + s];
    const int o = b.shell_ao[s0 + s], no = 2 * pi_(pi_tab, DXTB_I_L + t) + 1;
    double v = 0.0;
    for (int k = 0; k < no; ++k) v += q[o0 + o + k];
    qsh[s] = v;
    const double h = pf(pf_, DXTB_P_LGAM + t) * pf(pf_, DXTB_P_GAM + b.numbers[a0 + at]) + kEps;
    hard[s] = avg_kind == 0 ? 1.0 / h : h;
    if (s == 0 || b.shell_atom[s0 + s - 1] != at) sfirst[at] = s;
    if (s == nsh - 1) sfirst[nat] = nsh;
  }
  __syncthreads();
  const double gexp = pf(pf_, DXTB_P_SCAL + DXTB_S_GEXP);
  const double kexp = pf(pf_, DXTB_P_SCAL + DXTB_S_REP_KEXP);
  const double klight = pf(pf_, DXTB_P_SCAL + DXTB_S_REP_KLIGHT);
  const double rcut = pf(pf_, DXTB_P_SCAL + DXTB_S_REP_CUTOFF);
  const double dmp3 = pf(pf_, DXTB_P_SCAL + DXTB_S_DMP3), dmp5 = pf(pf_, DXTB_P_SCAL + DXTB_S_DMP5);
  for (int i = first + w; i < min(first + kGradAtoms, nat); i += (int)(blockDim.x >> 5)) {
    const double *pa = b.positions + 3 * (a0 + i);
    const int zi = b.numbers[a0 + i];
    double gi[3] = {0.0, 0.0, 0.0};
    double dmr_i = 0.0, qi = 0.0;
    for (int s = sfirst[i]; s < sfirst[i + 1]; ++s) qi += qsh[s];
    // d/dR_i of every ordered pair (i, j) and (j, i)
    for (int j = lane; j < nat; j += 32) {
      if (j == i) continue;
      const double *pb = b.positions + 3 * (a0 + j);
      const int zj = b.numbers[a0 + j];
      const double r[3] = {pa[0] - pb[0], pa[1] - pb[1], pa[2] - pb[2]};
      const double R = sqrt(r[0] * r[0] + r[1] * r[1] + r[2] * r[2]);
      double dEdR = 0.0, qj = 0.0;
      // ES2 (coulomb/secondorder.py:799-872): E = 1/2 q gamma q
      const double re = R + kEps;
      const double dg = gexp == 2.0 ? re * re : pow(re, gexp);
      const double dre = gexp == 2.0 ? re : pow(re, gexp - 1.0);
      for (int sj = sfirst[j]; sj < sfirst[j + 1]; ++sj) {
        const double hj = hard[sj];
        double v = 0.0;
        for (int si = sfirst[i]; si < sfirst[i + 1]; ++si) {
          const double hi = hard[si];
          double iavg;  // inverse of the averaged hardness
          if (avg_kind == 0) iavg = 0.5 * (hi + hj);
          else if (avg_kind == 1) iavg = 2.0 / (hi + hj);
          else iavg = 1.0 / sqrt(hi * hj);
          const double tmp = dg + (gexp == 2.0 ? iavg * iavg : pow(iavg, gexp));
          const double dgam = gexp == 2.0 ? dre / (tmp * sqrt(tmp)) : pow(tmp, -1.0 / gexp - 1.0) * dre;
          v += qsh[si] * dgam;  // both orderings: 2 * 1/2
        }
        dEdR -= qsh[sj] * v;
        qj += qsh[sj];
      }
      // repulsion (classicals/repulsion/base.py:351-430)
      if (R <= rcut) {
        const double a = sqrt(pf(pf_, DXTB_P_AREP + zi) * pf(pf_, DXTB_P_AREP + zj) + kTiny);
        const double k = (klight >= 0.0 && zi <= 2 && zj <= 2) ? klight : kexp;
        const double rk = pow_p(R, k);
        const double e = pf(pf_, DXTB_P_ZEFF + zi) * pf(pf_, DXTB_P_ZEFF + zj) * exp(-a * rk) / R;
        dEdR += -(a * rk * k + 1.0) * e / R;
      }
      for (int x = 0; x < 3; ++x) gi[x] += dEdR * r[x] / R;
      // AES2 pair terms e_ij + e_ji (coulomb/multipole.py:373-640)
      if (multipole) {
        const double M = 0.5 * (mrad[a0 + i] + mrad[a0 + j]);
        const double rr = M / R;
        const double r3d = pow_p(rr, dmp3), r5d = pow_p(rr, dmp5);
        const double f3 = 1.0 / (1.0 + 6.0 * r3d), f5 = 1.0 / (1.0 + 6.0 * r5d);
        const double df3 = f3 * f3 * 6.0 * dmp3 * r3d / R, df5 = f5 * f5 * 6.0 * dmp5 * r5d / R;
        const double df3M = -f3 * f3 * 6.0 * dmp3 * r3d / M, df5M = -f5 * f5 * 6.0 * dmp5 * r5d / M;
        const double iR = 1.0 / R, iR3 = iR * iR * iR, iR5 = iR3 * iR * iR;
        const double h3 = iR3 * f3, dh3 = -3.0 * iR3 * iR * f3 + iR3 * df3;
        const double dk3 = -3.0 * iR3 * iR * f5 + iR3 * df5;  // d/dR of k3 = f5 / R^3
        const double k5 = iR5 * f5, dk5 = -5.0 * iR5 * iR * f5 + iR5 * df5;
        double gr[3] = {0.0, 0.0, 0.0};
        double dM = 0.0;
        // two orderings: (i, j) with vector r and (j, i) with -r
        for (int ord = 0; ord < 2; ++ord) {
          const int I = ord == 0 ? i : j, J = ord == 0 ? j : i;
          const double sgn = ord == 0 ? 1.0 : -1.0;
          const double rv[3] = {sgn * r[0], sgn * r[1], sgn * r[2]};
          const double qI = (ord == 0 ? qi : qj);
          const double *u = dp + 3 * (a0 + J), *av = dp + 3 * (a0 + I);
          const double *wq = qp + 6 * (a0 + J);
          const double ru = rv[0] * u[0] + rv[1] * u[1] + rv[2] * u[2];
          const double ra = rv[0] * av[0] + rv[1] * av[1] + rv[2] * av[2];
          const double ab = av[0] * u[0] + av[1] * u[1] + av[2] * u[2];
          const double Wm[3][3] = {{wq[0], wq[1], wq[3]}, {wq[1], wq[2], wq[4]}, {wq[3], wq[4], wq[5]}};
          double Wr[3];
          for (int x = 0; x < 3; ++x) Wr[x] = Wm[x][0] * rv[0] + Wm[x][1] * rv[1] + Wm[x][2] * rv[2];
          const double rWr = rv[0] * Wr[0] + rv[1] * Wr[1] + rv[2] * Wr[2];
          double gv[3];
          for (int x = 0; x < 3; ++x) {
            // A: q_I (r.u) h3
            double v = qI * (u[x] * h3 + ru * dh3 * rv[x] * iR);
            // B: 1/2 [(a.b) k3 - 3 (r.a)(r.b) k5]
            v += 0.5 * (ab * dk3 * rv[x] * iR - 3.0 * (av[x] * ru + u[x] * ra) * k5 -
                        3.0 * ra * ru * dk5 * rv[x] * iR);
            // C: q_I (r W r) k5
            v += qI * (2.0 * Wr[x] * k5 + rWr * dk5 * rv[x] * iR);
            gv[x] = v;
          }
          // d e / d r (r = R_I - R_J); atom i gets +gv for ord 0, -gv for ord 1 (r = R_j - R_i)
          for (int x = 0; x < 3; ++x) gr[x] += sgn * gv[x];
          dM += qI * ru * iR3 * df3M + 0.5 * (ab * iR3 - 3.0 * ra * ru * iR5) * df5M + qI * rWr * iR5 * df5M;
        }
        for (int x = 0; x < 3; ++x) gi[x] += gr[x];
        dmr_i += 0.5 * dM;  // e_ij and e_ji both depend on M = (m_i + m_j) / 2
      }
    }
#pragma unroll
    for (int x = 0; x < 3; ++x) gi[x] = warp_sum(gi[x]);
    dmr_i = warp_sum(dmr_i);
    if (lane == 0) {
      for (int x = 0; x < 3; ++x) atomicAdd(&grad[3 * (a0 + i) + x], gi[x]);
      if (multipole) {
        // AES2 damping radius -> dE/dCN (coulomb/multipole.py:330-335)
        const double kx = pf(pf_, DXTB_P_SCAL + DXTB_S_MP_KEXP), sh = pf(pf_, DXTB_P_SCAL + DXTB_S_MP_SHIFT);
        const double rmax = pf(pf_, DXTB_P_SCAL + DXTB_S_MP_RMAX);
        const double rad = pf(pf_, DXTB_P_MPRAD + zi), vcn = pf(pf_, DXTB_P_MPVCN + zi);
        const double t1 = exp(-kx * (cn[a0 + i] - vcn - sh));
        const double dmdcn = (rmax - rad) * kx * t1 / ((1.0 + t1) * (1.0 + t1));
        atomicAdd(&dedcn[a0 + i], dmr_i * dmdcn);
      }
    }
  }
}

// Everything before the coordination-number chain rule, except pairs with a d
// shell: the first npb CTAs take shell pairs, `per` <= 32 a warp at a time (s-s
// and s-p 32 / per lanes each, then the p-p ones two at once), the others kGradAtoms
// atoms of a molecule. All is bound by the FP64 pipe; one launch fills the SMs
// to the end, where three left a tail each.
template <int NC>
__global__ void __launch_bounds__(128)
    k_grad_terms(dxtb_batch b, const double *__restrict__ pf_, const int32_t *__restrict__ pi_tab,
                 const double *__restrict__ cn, const double *__restrict__ mrad, const double *__restrict__ P,
                 const double *__restrict__ W, const double *__restrict__ S, const double *__restrict__ D,
                 const double *__restrict__ q, const double *__restrict__ dp, const double *__restrict__ qp,
                 const double *__restrict__ vorb, const double *__restrict__ vdp, const double *__restrict__ vqp,
                 double *__restrict__ dedcn, double *__restrict__ grad, int npb, int per, ClassFilter flt) {
  extern __shared__ double sm[];
  __shared__ double s_es[4][2][9 * NC];
  if ((int)blockIdx.x >= npb) {
    const int groups = (b.max_nat + kGradAtoms - 1) / kGradAtoms, r = (int)blockIdx.x - npb;
    const int m = r / groups;
    if (!in_class(flt, b, m)) return;
    grad_atoms(b, pf_, pi_tab, cn, mrad, q, dp, qp, NC > 1, dedcn, grad, m, (r % groups) * kGradAtoms, sm);
    return;
  }
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, nsub = 32 / per, part = lane % nsub;
  const int64_t npairs = b.pair_off[b.nmol];
  for (int64_t k0 = ((int64_t)blockIdx.x * 4 + w) * per; k0 < npairs; k0 += (int64_t)npb * 4 * per) {
    GPair g = {};
    int kind = 0;  // 1: s-s or s-p, 2: p-p
    const int64_t k = k0 + lane / nsub;
    if (k < npairs) {
      shell_pair(b, k, g.m, g.i, g.j);
      if (in_class(flt, b, g.m)) {
        const int64_t s0 = b.shell_off[g.m];
        const int la = pi_(pi_tab, DXTB_I_L + b.shell_type[s0 + g.i]);
        const int lb = pi_(pi_tab, DXTB_I_L + b.shell_type[s0 + g.j]);
        kind = la > 1 || lb > 1 ? 0 : (la + lb <= 1 ? 1 : 2);
        if (kind == 1 && la == 1) {  // evaluate the s-p mirror: the s shell on the bra
          const int x = g.i;
          g.i = g.j;
          g.j = x;
        }
      }
    }
    GScale sc = {};
    double ps = 0.0, gr[3] = {0.0, 0.0, 0.0};
    if (kind == 1) {
      grad_pair_setup(b, pi_tab, g);
      if (g.lb == 0)
        grad_pair_sp<0, NC>(b, pf_, pi_tab, cn, P, W, S, D, vorb, vdp, vqp, g, part, nsub, sc, ps, gr);
      else
        grad_pair_sp<1, NC>(b, pf_, pi_tab, cn, P, W, S, D, vorb, vdp, vqp, g, part, nsub, sc, ps, gr);
    }
    for (int o = 1; o < nsub; o <<= 1)
#pragma unroll
      for (int x = 0; x < 3; ++x) gr[x] += __shfl_xor_sync(0xffffffffu, gr[x], o);
    if (kind == 1 && part == 0) {
      grad_add_cn(pf_, g, sc, ps, dedcn);
      if (g.ai != g.aj) grad_add(g, sc, ps, gr, grad);
    }
    unsigned todo = __ballot_sync(0xffffffffu, kind == 2 && part == 0);
    while (todo != 0) {
      const int l0 = __ffs(todo) - 1;
      todo &= todo - 1;
      const int l1 = todo != 0 ? __ffs(todo) - 1 : -1;
      todo &= todo - 1;
      const bool active = lane < 16 || l1 >= 0;
      const int src = lane < 16 || l1 < 0 ? l0 : l1;
      GPair h;
      h.m = __shfl_sync(0xffffffffu, g.m, src);
      h.i = __shfl_sync(0xffffffffu, g.i, src);
      h.j = __shfl_sync(0xffffffffu, g.j, src);
      grad_pair_setup(b, pi_tab, h);
      grad_pair_pp<NC>(b, pf_, pi_tab, cn, P, W, S, D, vorb, vdp, vqp, dedcn, grad, h, active, s_es[w][lane >> 4]);
      __syncwarp();  // the next pairs reuse the coefficients' memory
    }
  }
}

// Coordination-number chain rule (tad_mctc cn_d3 restated), after all of dedcn:
// a warp per atom.
__global__ void __launch_bounds__(128)
    k_grad_cn(dxtb_batch b, const double *__restrict__ pf_, const int32_t *__restrict__ pi_tab,
              const double *__restrict__ dedcn, double *__restrict__ grad, ClassFilter flt) {
  const int groups = (b.max_nat + kGradAtoms - 1) / kGradAtoms;
  const int m = (int)blockIdx.x / groups, first = ((int)blockIdx.x % groups) * kGradAtoms;
  if (!in_class(flt, b, m)) return;
  const int64_t a0 = b.atom_off[m];
  const int nat = (int)(b.atom_off[m + 1] - a0), lane = threadIdx.x & 31;
  const int cn_kind = pi_(pi_tab, DXTB_I_SCAL + DXTB_IS_CN_KIND);
  const double cutoff = pf(pf_, DXTB_P_SCAL + DXTB_S_CN_CUTOFF);
  for (int i = first + (int)(threadIdx.x >> 5); i < min(first + kGradAtoms, nat); i += (int)(blockDim.x >> 5)) {
    const double *pa = b.positions + 3 * (a0 + i);
    const double rci = pf(pf_, DXTB_P_RCOV + b.numbers[a0 + i]);
    const double di = dedcn[a0 + i];
    double gi[3] = {0.0, 0.0, 0.0};
    for (int j = lane; j < nat; j += 32) {
      if (j == i) continue;
      const double *pb = b.positions + 3 * (a0 + j);
      const double r[3] = {pa[0] - pb[0], pa[1] - pb[1], pa[2] - pb[2]};
      const double R = sqrt(r[0] * r[0] + r[1] * r[1] + r[2] * r[2]);
      if (R > cutoff) continue;
      const double r0 = rci + pf(pf_, DXTB_P_RCOV + b.numbers[a0 + j]);
      double dc;
      if (cn_kind == 0) {
        exp_count_d(R, r0, 16.0, &dc);
      } else {
        double d1, d2;
        const double c1 = exp_count_d(R, r0, 10.0, &d1);
        const double c2 = exp_count_d(R, r0 + 2.0, 20.0, &d2);
        dc = d1 * c2 + c1 * d2;
      }
      const double f = (di + dedcn[a0 + j]) * dc / R;
      for (int x = 0; x < 3; ++x) gi[x] += f * r[x];
    }
#pragma unroll
    for (int x = 0; x < 3; ++x) gi[x] = warp_sum(gi[x]);
    if (lane == 0)
      for (int x = 0; x < 3; ++x) atomicAdd(&grad[3 * (a0 + i) + x], gi[x]);
  }
}

}  // namespace dxtb

using namespace dxtb;

constexpr int kTermsSmem = 220 * 1024;  // 2 nsh + nat / 2 doubles: as many atoms as 200 KB of nsh + 3 nat
constexpr size_t gSmem = sizeof(double) * gWarps * (gChunk * gTab + 2 * gNComp * 36);

namespace dxtb {

int32_t launch_gradient(const dxtb_batch *b, const double *par_f, const int32_t *par_i,
                        const double *cn, const double *mrad, const double *density,
                        const double *wdensity, const double *q, const double *dp, const double *qp,
                        const double *vorb, const double *vdp, const double *vqp,
                        const double *overlap, const double *dipole, double *dedcn, double *grad,
                        const ClassFilter &f, cudaStream_t st) {
  if (!b || b->nmol <= 0 || !cn || !density || !wdensity || !q || !vorb || !overlap || !dedcn ||
      !grad)
    return DXTB_ERR_ARGS;
  // The multipole (GFN2) terms are taken iff the dipole integrals are given.
  const int multipole = dipole != nullptr;
  if (multipole && (!vdp || !vqp || !dp || !qp || !mrad)) return DXTB_ERR_ARGS;
  static PerDeviceOnce attr;
  if (per_device_once(attr, [] {
        return cudaFuncSetAttribute(k_grad_pairs, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)gSmem) == cudaSuccess &&
               cudaFuncSetAttribute(k_grad_terms<1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    kTermsSmem) == cudaSuccess &&
               cudaFuncSetAttribute(k_grad_terms<gNComp>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    kTermsSmem) == cudaSuccess;
      }) != DXTB_OK)
    return DXTB_ERR_LAUNCH;
  const int64_t bound = (int64_t)b->nmol * b->max_nsh * (b->max_nsh + 1) / 2;
  const int groups = (b->max_nat + kGradAtoms - 1) / kGradAtoms;
  const size_t smem = sizeof(double) * (size_t)(2 * b->max_nsh + b->max_nat / 2 + 2);
  if (smem > kTermsSmem) return DXTB_ERR_TOO_LARGE;
  const auto terms = multipole ? k_grad_terms<gNComp> : k_grad_terms<1>;
  int sms = 0;
  if (device_sms(&sms) != DXTB_OK) return DXTB_ERR_LAUNCH;
  // pairs with a d shell: a warp each
  const int64_t dblocks = max((int64_t)1, min((bound + gWarps * kGradChunk - 1) / (gWarps * kGradChunk), (int64_t)sms * 16));
  k_grad_pairs<<<(unsigned)dblocks, gWarps * 32, gSmem, st>>>(*b, par_f, par_i, cn, density, wdensity, overlap,
                                                              dipole, vorb, vdp, vqp, multipole, dedcn, grad, f);
  DXTB_CHECK_LAUNCH();
  // few pairs: fewer of them a warp, more warps, several lanes for each
  int per = 32;
  while (per > 4 && bound < (int64_t)sms * 16 * per) per /= 2;
  const int npb = (int)max((int64_t)1, min((bound + 4 * per - 1) / (4 * per), (int64_t)sms * 16));
  const int64_t nblocks = npb + (int64_t)b->nmol * groups;
  if (nblocks > INT32_MAX) return DXTB_ERR_TOO_LARGE;
  terms<<<(unsigned)nblocks, 128, smem, st>>>(*b, par_f, par_i, cn, mrad, density, wdensity, overlap, dipole, q, dp,
                                              qp, vorb, vdp, vqp, dedcn, grad, npb, per, f);
  DXTB_CHECK_LAUNCH();
  k_grad_cn<<<(unsigned)(b->nmol * groups), 128, 0, st>>>(*b, par_f, par_i, dedcn, grad, f);
  DXTB_CHECK_LAUNCH();
  return DXTB_OK;
}

}  // namespace dxtb

extern "C" int32_t dxtb_gradient(const dxtb_batch *b, const double *par_f, const int32_t *par_i,
                                 const double *cn, const double *cn_mp, const double *mrad,
                                 const double *density, const double *wdensity, const double *q,
                                 const double *dp, const double *qp, const double *vorb,
                                 const double *vdp, const double *vqp, const double *overlap,
                                 const double *dipole, const double *unused0,
                                 const double *unused1, double *dedcn, double *dedcn_mp,
                                 double *grad, void *stream) {
  (void)cn_mp;
  (void)unused0;
  (void)unused1;
  (void)dedcn_mp;
  ClassFilter all;
  for (int c = 0; c < kClasses; ++c) all.thr[c] = 0;
  all.cls = -1;
  return launch_gradient(b, par_f, par_i, cn, mrad, density, wdensity, q, dp, qp, vorb, vdp, vqp,
                         overlap, dipole, dedcn, grad, all, (cudaStream_t)stream);
}

// qk_poles.cuh -- the FP64 pole sums of the diagonal GW self-energy for a tile of orbitals.
//
//   Sigma_p = sum_{q,m} 2 rho_pqm^2 g(w_p - e_q +- Om_m)  (+ for occupied q, - for virtual q)
//
// with its derivative and its occupied part (RGW_self_energy_diag.f90:44-84 and, for the SRG
// weights, RGW_SRG_self_energy_diag.f90).  Used by the workspace entry points (k_sigma.cu) and by
// the allocation-free one (k_noalloc.cu).
//
// What bounds it: the FP64 pipe (about two lanes per SM and clock), not memory: a term reads 8
// bytes and costs 8 to 10 FP64 instructions.  Hence
//  - lanes = excitations m, a warp's tile = 8 orbitals p of one q: the eight w_p - e_q are formed
//    once, by eight lanes, for all of the warp's terms, and a warp whose orbitals are few (the last ones of a Newton search) does
//    only their work.  The 8 loads of a lane walk along one 64-byte piece of rho, so every sector
//    is read once although the lanes are N^2 apart;
//  - one cubic Newton step for the reciprocal (3 instructions) instead of two quadratic ones (4),
//    range checks on the integer pipe, the factor 2 applied to the sums, and
//    (eps^2 - eta^2)/(eps^2 + eta^2) = 1 - 2 eta^2/(eps^2 + eta^2);
//  - SRG: 1 - exp(-2 s eps^2) is exactly 1 in FP64 once 2 s eps^2 >= 38 (exp(-38) < 2^-54).  Om
//    being ascending, the poles near w are neighbouring lanes, so few warps evaluate an exp at all.
// Measured (N = 150, nS = 2489, 56M terms, eta = 0.05): 1.97 ms with lanes = orbitals and 20 FP64
// instructions a term, 1.14 ms like this; its instructions alone take 0.98 ms at two a clock and
// SM.  N = 200, nS = 3600: 6.3 -> 2.9 ms a sweep; SRG at N = 120, s = 500: 2.0 -> 0.50 ms.
#pragma once
#include "qk_internal.cuh"

namespace qk_poles {

constexpr int PT = 8;      // orbitals per tile
constexpr int WARPS = 8;   // warps split the q of a CTA's range
enum { KIND_ETA0 = 0, KIND_ETA = 1, KIND_SRG = 2 };

// 1/x as qk_rcp3, with the range check on the high word alone ([2^-996, 2^996) here; with both words it
// cost 10 % of the sweep)
__device__ __forceinline__ double rcp3(double x) {
  const unsigned h = (unsigned)__double2hiint(x) & 0x7fffffffu;
  if (h - 0x01B00000u >= 0x7E300000u - 0x01B00000u) return 1.0 / x;
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  const double e = __fma_rn(-x, r, 1.0);
  return __fma_rn(r, __fma_rn(e, e, e), r);
}

// one term: s += x^2 g(eps), d -= x^2 g'(eps)
//   eta: c0 = eta^2, c1 = -2 eta^2.   SRG: c1 = -2 flow, hthr = high word of sqrt(19 / flow)
template <int KIND>
__device__ __forceinline__ void term(double x, double eps, double c0, double c1, unsigned hthr,
                                     double& s, double& d) {
  const double x2 = __dmul_rn(x, x);
  if (KIND == KIND_ETA) {
    const double rr = rcp3(__fma_rn(eps, eps, c0));
    const double t = __dmul_rn(x2, rr);
    s = __fma_rn(t, eps, s);
    d = __fma_rn(t, __fma_rn(rr, c1, 1.0), d);
  } else {
    const double ir = rcp3(eps);
    double t = __dmul_rn(x2, ir);
    if (KIND == KIND_SRG) {
      if (((unsigned)__double2hiint(eps) & 0x7fffffffu) <= hthr)
        t = __dmul_rn(__dmul_rn(x2, 1.0 - exp(c1 * eps * eps)), ir);
    }
    s = __dadd_rn(s, t);
    d = __fma_rn(t, ir, d);
  }
}

// sums of v[0..7] over the warp; the lane with lane & 3 == 0 gets that of v[lane >> 2].  The tree
// is the same for all eight, so an orbital's sum does not depend on its place in the tile.
__device__ __forceinline__ double reduce8(const double (&v)[PT], int lane) {
  double a[4], b[2], c;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const bool up = lane & 16;
    const double give = up ? v[i] : v[i + 4], keep = up ? v[i + 4] : v[i];
    a[i] = keep + __shfl_xor_sync(0xffffffffu, give, 16);
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const bool up = lane & 8;
    const double give = up ? a[i] : a[i + 2], keep = up ? a[i + 2] : a[i];
    b[i] = keep + __shfl_xor_sync(0xffffffffu, give, 8);
  }
  {
    const bool up = lane & 4;
    const double give = up ? b[0] : b[1], keep = up ? b[1] : b[0];
    c = keep + __shfl_xor_sync(0xffffffffu, give, 4);
  }
  c += __shfl_xor_sync(0xffffffffu, c, 2);
  c += __shfl_xor_sync(0xffffffffu, c, 1);
  return c;
}

struct Tile {
  int p[PT];        // orbitals of the tile
  double w[PT];     // their evaluation energies
  double red[3][WARPS][PT];
};

struct Range {
  int N, nO;
  int q0, q1;       // q range of the CTA
  int m0, m1;       // m range of the CTA
};

// adds the terms of the virtual (VIR) or occupied q of [qa, qb) to s, d; the warps take q in turn,
// beginning with warp rot
template <int KIND, bool VIR>
__device__ __forceinline__ void sweep(const Tile& T, int np, const Range& g, int qa, int qb, int rot,
                                      const double* __restrict__ e, const double* __restrict__ Om,
                                      const double* __restrict__ rho, double c0, double c1,
                                      unsigned hthr, double (&s)[PT], double (&d)[PT]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long N1 = g.N, N2 = N1 * N1;
  const double wl = T.w[(lane & (PT - 1)) < np ? lane & (PT - 1) : 0];
  for (int mb = g.m0; mb < g.m1; mb += 32) {
    const int m = mb + lane;
    const bool ok = m < g.m1;
    // lanes past the end take a zero amplitude at a pole far away
    const double om = ok ? __ldg(Om + m) : 1e30;
    const double* r = rho + N2 * (ok ? m : g.m0);
    for (int q = qa + ((warp - rot) & (WARPS - 1)); q < qb; q += WARPS) {
      double x[PT];
#pragma unroll
      for (int j = 0; j < PT; ++j) x[j] = (ok && j < np) ? __ldg(r + N1 * q + T.p[j]) : 0.0;
      const double c = wl - __ldg(e + q);
#pragma unroll
      for (int j = 0; j < PT; ++j)
        if (j < np) {
          const double cj = __shfl_sync(0xffffffffu, c, j);
          term<KIND>(x[j], VIR ? cj - om : cj + om, c0, c1, hthr, s[j], d[j]);
        }
    }
  }
}

// the CTA's partial sums for the np <= 8 orbitals of T (filled and synchronised by the caller):
// part[p] = sum, part[stride + p] = derivative, part[2 stride + p] = occupied part of the sum
template <int KIND>
__device__ __forceinline__ void tile_sums(Tile& T, int np, const Range& g,
                                          const double* __restrict__ e,
                                          const double* __restrict__ Om,
                                          const double* __restrict__ rho, double eta, double flow,
                                          double* __restrict__ part, size_t stride) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const double c0 = eta * eta, c1 = KIND == KIND_SRG ? -2.0 * flow : -2.0 * c0;
  // a flow that is not positive gives the high word of an infinity or a NaN: always the exp, but for
  // |eps| from 2^98 on, where only the padding lanes' 1e30 lies (their zero amplitude times 1 - exp of
  // a large positive number, with a negative flow, would be a NaN)
  const unsigned hthr =
      KIND == KIND_SRG
          ? min((unsigned)__double2hiint(sqrt(19.0 / flow)) & 0x7fffffffu, (1023u + 98u) << 20)
          : 0u;
  double s[PT], d[PT];
#pragma unroll
  for (int j = 0; j < PT; ++j) s[j] = d[j] = 0.0;
  const int qo = min(g.q1, max(g.q0, g.nO));  // first virtual q of the range
  sweep<KIND, false>(T, np, g, g.q0, qo, 0, e, Om, rho, c0, c1, hthr, s, d);
  const double so = reduce8(s, lane);
#pragma unroll
  for (int j = 0; j < PT; ++j) s[j] = 0.0;
  sweep<KIND, true>(T, np, g, qo, g.q1, qo - g.q0, e, Om, rho, c0, c1, hthr, s, d);
  const double sv = reduce8(s, lane), ds = reduce8(d, lane);
  if ((lane & 3) == 0) {
    T.red[0][warp][lane >> 2] = so;
    T.red[1][warp][lane >> 2] = sv;
    T.red[2][warp][lane >> 2] = ds;
  }
  __syncthreads();
  if (threadIdx.x < np) {
    double o = 0.0, v = 0.0, dd = 0.0;
    for (int k = 0; k < WARPS; ++k) {
      o += T.red[0][k][threadIdx.x];
      v += T.red[1][k][threadIdx.x];
      dd += T.red[2][k][threadIdx.x];
    }
    const int p = T.p[threadIdx.x];
    part[p] = 2.0 * (o + v);
    part[stride + p] = -2.0 * dd;
    part[2 * stride + p] = 2.0 * o;
  }
}

// Sig = sum of the chunks' partials, Z = 1/(1 - derivative); returns the caller's lane-0 share of
// the occupied parts of the virtual p (0 on the other lanes).  One block; a warp per orbital.
__device__ __forceinline__ double final_sums(int N, int nC, int nO, int nR, int nchunks,
                                             const double* __restrict__ part,
                                             double* __restrict__ Sig, double* __restrict__ Z) {
  const size_t stride = (size_t)nchunks * N;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  double gm = 0.0;
  for (int p = warp; p < N; p += nw) {
    double s = 0.0, d = 0.0, o = 0.0;
    if (p >= nC && p < N - nR) {
      for (int c = lane; c < nchunks; c += 32) {
        s += part[(size_t)c * N + p];
        d += part[(size_t)c * N + p + stride];
        o += part[(size_t)c * N + p + 2 * stride];
      }
      for (int k = 16; k > 0; k >>= 1) {
        s += __shfl_xor_sync(0xffffffffu, s, k);
        d += __shfl_xor_sync(0xffffffffu, d, k);
        o += __shfl_xor_sync(0xffffffffu, o, k);
      }
    }
    if (lane == 0) {
      Sig[p] = s;
      Z[p] = 1.0 / (1.0 - d);
      if (p >= nO) gm += o;
    }
  }
  return gm;
}

}  // namespace qk_poles

// k_tri_fx.cu -- Householder tridiagonalisation in 64-bit fixed point on the integer pipe: matrices up
// to order 615 resident in the shared memory of one thread-block cluster (k_tri_fx), larger ones by
// the whole grid (k_tri_fx_grid, further down).
//
// The FP64 tier's reduction of a Casida matrix (dsyev's dsytrd step) for the sizes that fit.  The
// grid-wide FP64 kernel (k_sytrd) pays ~10 us per column whatever the size -- a grid barrier, L2 round
// trips and FP64 block sums at 64 cycles per warp instruction.  Here
//   - A is full (not only its lower triangle) and row-cyclic over the cluster's CTAs, so row r's
//     part of p = A v is one warp's dot product and nothing is summed across CTAs;
//   - p_r and the next column's element A_(r,j+1) go to every CTA by one distributed-shared-memory
//     store instruction per row, and one cluster barrier (~0.25 us) ends the column;
//   - the arithmetic is fixed point: orthogonal similarity keeps |A_ij| <= ||A||_2, so with the matrix
//     scaled by the power of two S that makes min(||A||_inf, ||A||_F) / S < 1/2 an element is an int64 multiple of
//     2^-62, and a product of two such numbers is three 32 x 32 -> 64 multiply-adds (2 cycles per
//     warp each, against 64 for an FP64 FMA).  An element costs ~45 issue slots per column.
// Accuracy: every update rounds to 2^-62 S without bias; FP64 rounds to
// 2^-53 of the element.  The reflectors are normalised to unit length to ~2^-60, so the transformation
// is orthogonal to working precision, and the factorisation is backward stable with a smaller
// constant than in FP64 (the test measures both).  Elements below 2^-62 S are lost, which is why
// qk_dsyev_dev, which takes any matrix, stays with the FP64 kernel.  Integer sums make the result
// independent of the number of CTAs and of the order of summation.
//
// Column j (u = the previous reflector, |u| = 1, H = I - 2 u u^T):
//   K = u^T p;  w = p - K u;  x = column j of A - 2 (u w^T + w u^T);  d_j = x_j;
//   u' = unit vector of x_(j+1..) + sign(alpha) |x| e_1, e_j = -sign(alpha) |x|   (dlarfg's choice)
//   rows r > j: A_r -= 2 (u_r w + w_r u), p'_r = A_r u', broadcast p'_r and A_(r,j+1).
// Measured (one GB300), eigenvalues alone (this kernel plus the bisection), before -> now: n = 48
// 0.77 -> 0.30 ms, 128 1.84 -> 0.59, 256 3.55 -> 1.2, 400 5.55 -> 2.04, 600 8.43 -> 3.9.  Cycles of a
// column at n = 400 (48): K 0.8k (0.75k), w and x 0.4k (0.1k), the norm's sums and the reflector 1.5k
// (1.7k), u' 0.3k (0.1k), the rows 2.6k (2.0k), the cluster barrier with its wait 1.7k (1.1k), of
// which the release of the remote stores is about 0.9k.  The O(n) loops are kept rolled: unrolled by
// the compiler they cost 2 to 3 % (a thread runs them once or twice).  Tried and not kept: K from the
// row pass by remote stores (K 0.55k, but the rows 0.6k more), three and four rows of a warp at a time.
#include <cooperative_groups.h>
#include <mutex>
#include "qk_internal.cuh"

namespace cg = cooperative_groups;

namespace {

constexpr int WORKERS = 512;             // worker threads; one more warp writes d, e, tau and V
constexpr int VT = 256, VW = VT / 32;    // of them the O(n) vector work of a column
constexpr int THREADS = WORKERS + 32;
constexpr int NWARPS = WORKERS / 32;
constexpr int MAX_CL = 16;
constexpr int SMEM_MAX = 226 * 1024;

struct FxGroup {
  qk_tri_fx_args req[QK_TRI_FX_GROUP];
};

// x = h 2^32 + l' with l' signed; l = l' >> 1 (31 bits): in Q62, x = h 2^-30 + l 2^-61
struct Fx {
  int h, l;
};
__device__ __forceinline__ Fx fx_split(long long x) {
  const int lo = (int)(unsigned)x;
  return Fx{(int)(x >> 32) + (int)((unsigned)lo >> 31), lo >> 1};
}
__device__ __forceinline__ long long wide(int a, int b) { return (long long)a * b; }
constexpr long long CR_HALF = 1ll << 28;
// round(x y 2^62): the l l term (zero mean, below 2^-62) is dropped
__device__ __forceinline__ long long fx_mul(Fx x, Fx y) {
  const long long hh = wide(x.h, y.h);
  const long long cr = CR_HALF + wide(x.h, y.l) + wide(x.l, y.h);
  return (hh << 2) + (cr >> 29);
}
// 2 (a b + c d)
__device__ __forceinline__ long long fx_mul2(Fx a, Fx b, Fx c, Fx d) {
  const long long hh = wide(a.h, b.h) + wide(c.h, d.h);
  const long long cr =
      (CR_HALF >> 1) + wide(a.h, b.l) + wide(a.l, b.h) + wide(c.h, d.l) + wide(c.l, d.h);
  return (hh << 3) + (cr >> 28);
}
// the same with the l l term (its upper 29 bits): without it every product errs by 0.3 x 2^-62, which
// over the thousands of products of a long row outweighs the rounding
__device__ __forceinline__ long long ll_term(int a, int b) { return wide(a >> 16, b >> 15); }
__device__ __forceinline__ long long fx_mul2x(Fx a, Fx b, Fx c, Fx d) {
  const long long hh = wide(a.h, b.h) + wide(c.h, d.h);
  const long long cr = (CR_HALF >> 1) + wide(a.h, b.l) + wide(a.l, b.h) + wide(c.h, d.l) +
                       wide(c.l, d.h) + ll_term(a.l, b.l) + ll_term(c.l, d.l);
  return (hh << 3) + (cr >> 28);
}
constexpr long long FX_ONE = 1ll << 62;

// 1 / sqrt(4 m4) for m4 in [1/4, 1]: the hardware's FP32 value r0 (an integer of Q30, relative error
// below 2^-21) and one third-order step r = r0 (1 + h + 3 h^2 / 2), h = (1 - 4 m4 r0^2) / 2
__device__ __forceinline__ long long fx_rsqrt4(long long m4) {
  const float m = (float)(int)(m4 >> 32) * 0x1p-28f;     // 4 m4 in [1, 4]
  const int r0 = (int)fminf(rsqrtf(m) * 0x1p30f, 0x1p30f);
  const long long u = fx_mul(fx_split(m4), fx_split(wide(r0, r0) << 2));  // m4 r0^2, near 1/4
  const long long h = ((FX_ONE >> 2) - u) << 1;                             // |h| < 2^42 (Q62)
  const int hq = (int)(h >> 20);                                           // Q42
  const long long c = h + ((3 * wide(hq, hq)) >> 23);                      // h + 3 h^2 / 2
  // r0 c: c in two parts of 25 + 18 bits
  const int ch = (int)(c >> 18), clow = (int)(c & 0x3FFFF);
  return ((long long)r0 << 32) + ((wide(r0, ch) + (wide(r0, clow) >> 18)) >> 12);
}

// double -> Q62 of the scaled matrix (x 2^(62 - E - 1)), 2^E above the norm bound
__device__ __forceinline__ long long fx_from_double(double x, int E) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const int ex = (int)((b >> 52) & 0x7FF);
  const unsigned long long m = (b & 0xFFFFFFFFFFFFFull) | (ex ? 1ull << 52 : 0ull);
  const int sh = max(ex, 1) - 1075 + 61 - E;
  long long q;
  if (sh >= 0) q = (long long)(m << min(sh, 63));
  else if (sh > -63) q = (long long)((m + (1ull << (-sh - 1))) >> -sh);
  else q = 0;
  return (long long)b < 0 ? -q : q;
}
__device__ __forceinline__ double pow2(int k) {  // |k| <= 1022
  return __longlong_as_double((long long)(k + 1023) << 52);
}
// x 2^k rounded to a double, on the integer pipe where the result is a normal number
__device__ __forceinline__ double fx_to_double(long long x, int k) {
  if (x == 0) return 0.0;
  unsigned long long m = (unsigned long long)(x < 0 ? -x : x);
  const int z = __clzll((long long)m);
  m <<= z;                                            // leading bit at 63
  const unsigned rem = (unsigned)m & 0x7FFu;
  m >>= 11;
  m += rem + (unsigned)(m & 1ull) > 0x400u ? 1ull : 0ull;
  const int ex = 63 - z + k + 1023;
  const unsigned long long sign = x < 0 ? 1ull << 63 : 0ull;
  if (ex > 0 && ex < 2046)
    return __longlong_as_double((long long)((((unsigned long long)(ex - 1) << 52) + m) | sign));
  const int q = max(-2200, min(2200, ex - 1023)), q1 = q / 3;
  return __longlong_as_double((long long)(((1022ull << 52) + m) | sign)) * pow2(q1) * pow2(q1) *
         pow2(q - 2 * q1);
}

// sum of one int64 per lane over the warp, in every lane (REDUX is 32 bits wide and issues slowly:
// three of them took 330 cycles with all warps at it, this butterfly ~150)
__device__ __forceinline__ long long warp_sum64(long long v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ void vec_bar() { asm volatile("bar.sync 1, 256;" ::: "memory"); }
__device__ __forceinline__ long long sum_parts(const long long* p) {
  long long t = 0;
#pragma unroll
  for (int w = 0; w < VW; ++w) t += p[w];
  return t;
}

struct Scal {             // one column's scalars, written by one thread
  long long f;            // u'_i = (x_i << sh) f
  long long u1;           // u'_(j+1), signed
  long long nx;           // |x| 2^(sh - xs)
  int sh;
  long long g;            // 1 / (2 |u1|)
  int neg, zero;          // alpha < 0; no reflector (x = 0, or the last column)
  long long dj, alpha;
};

// from the sums s0 of h^2 and s1 of h l' 2^-sq + l'^2 2^-(33 + sq): |x|^2 = s0 2^-60 + s1 2^(sq - 91)
__device__ __forceinline__ void reflector(long long s0, long long s1, int sq, int xs, bool last,
                                          long long xj, long long alpha, int lane, Scal& out) {
  Scal t;
  t.dj = xj;
  t.alpha = alpha;
  t.neg = alpha < 0;
  t.zero = xs < 0 || last;
  t.sh = 0;
  t.f = t.u1 = t.nx = t.g = 0;
  if (!t.zero) {
    // |x|^2 = T 2^(sq - 91): m4 = |x|^2 4^(sh - xs) in [1/4, 1)
    const int fb = 91 - sq;
    unsigned long long hi = (unsigned long long)(s0 >> (124 - fb)), lo = (unsigned long long)s0 << (fb - 60);
    const unsigned long long lo2 = lo + (unsigned long long)s1;
    hi += (unsigned long long)(s1 >> 63) + (lo2 < lo ? 1ull : 0ull);
    lo = lo2;
    const int lead = 128 - __clzll((long long)hi);        // bits of T (hi > 0)
    const int q = (fb - lead) >> 1;                       // T 4^q has fb - 1 or fb bits
    const int down = fb - 62 - 2 * q;                     // m4 (Q62) = T >> down, 0 < down < 64
    const long long m4 = (long long)((hi << (64 - down)) | (lo >> down));
    const long long r = fx_rsqrt4(m4);                    // 1 / (2 |x'|), |x'| = |x| 2^(q + xs)
    const Fx rs = fx_split(r);
    t.nx = fx_mul(fx_split(m4), rs) << 1;                 // |x'| in [1/2, 1)
    t.sh = q + xs;
    const long long ax = (alpha < 0 ? -alpha : alpha) << t.sh;
    // a = |alpha| / |x| in [0, 1]; b = (1 + a) / 2; u1 = sqrt(b); u_i = x_i / (2 |x| u1)
    long long b = (FX_ONE >> 1) + fx_mul(fx_split(ax), rs);
    b = b > FX_ONE ? FX_ONE : b;
    t.g = fx_rsqrt4(b);                                   // 1 / (2 sqrt(b))
    const Fx gs = fx_split(t.g);
    const long long u1 = fx_mul(fx_split(b), gs) << 1;
    t.u1 = alpha < 0 ? -u1 : u1;
    t.f = fx_mul(rs, gs) << 1;                            // 1 / (2 |x'| u1)
  }
  if (lane == 0) out = t;
}

// R own rows (lr, lr + NWARPS): the rank-2 update, the dot product with u' and the broadcast of p'
// and of the next column's element.  The loads of two column groups are issued together.
template <int R>
__device__ __forceinline__ void row_pass(long long* As, int lr, int n, int j, int CL, int rank, int par,
                                         int lane, const Fx* U, const Fx* Wb, const Fx* Un,
                                         long long* Pb, long long* Xb, cg::cluster_group& cl) {
  long long* Ar[R];
  Fx ur[R], wr[R];
  long long hh[R], cr[R], xn[R];
#pragma unroll
  for (int q = 0; q < R; ++q) {
    const int r = (lr + q * NWARPS) * CL + rank;
    Ar[q] = As + (size_t)(lr + q * NWARPS) * n;
    ur[q] = U[r];
    wr[q] = Wb[r];
    hh[q] = cr[q] = xn[q] = 0;
  }
  constexpr int B = 2;                     // column groups in flight
  for (int c0 = j + 1; c0 < n; c0 += 32 * B) {
    Fx u[B], w[B], v[B];
    long long y[R][B];
#pragma unroll
    for (int b = 0; b < B; ++b) {
      const int c = c0 + 32 * b + lane, cc = c < n ? c : n - 1;
      u[b] = U[cc];
      w[b] = Wb[cc];
      v[b] = Un[cc];
      if (c >= n) v[b] = Fx{0, 0};
#pragma unroll
      for (int q = 0; q < R; ++q) y[q][b] = Ar[q][cc];
    }
#pragma unroll
    for (int b = 0; b < B; ++b) {
      const int c = c0 + 32 * b + lane;
#pragma unroll
      for (int q = 0; q < R; ++q) {
        y[q][b] -= fx_mul2(ur[q], w[b], wr[q], u[b]);
        if (c < n) Ar[q][c] = y[q][b];
        const Fx ys = fx_split(y[q][b]);
        hh[q] += wide(ys.h, v[b].h);
        cr[q] += wide(ys.h, v[b].l) + wide(ys.l, v[b].h);
      }
    }
    if (c0 == j + 1) {
#pragma unroll
      for (int q = 0; q < R; ++q) xn[q] = y[q][0];
    }
  }
  long long p[R];
#pragma unroll
  for (int q = 0; q < R; ++q) p[q] = (hh[q] << 2) + ((cr[q] + CR_HALF) >> 29);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int q = 0; q < R; ++q) p[q] += __shfl_xor_sync(0xffffffffu, p[q], o);
  // lanes 0..15: p' to CTA lane, lanes 16..31: the next column's element to CTA lane - 16
  const int dst = lane & 15;
#pragma unroll
  for (int q = 0; q < R; ++q) {
    const long long x = __shfl_sync(0xffffffffu, xn[q], 0);
    if (dst < CL) {
      long long* base = (lane < 16 ? Pb : Xb) + (par ^ 1) * n + (lr + q * NWARPS) * CL + rank;
      *cl.map_shared_rank(base, dst) = lane < 16 ? p[q] : x;
    }
  }
}

// cluster b of the grid reduces matrix b
__global__ void __launch_bounds__(THREADS, 1) k_tri_fx(const __grid_constant__ FxGroup grp) {
  cg::cluster_group cl = cg::this_cluster();
  const int CL = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const qk_tri_fx_args& a = grp.req[blockIdx.x / CL];
  const int n = a.n, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rows = (n - rank + CL - 1) / CL;      // rows rank, rank + CL, ..
  const int max_rows = (n + CL - 1) / CL;
  extern __shared__ long long sm[];
  long long* As = sm;                                // rows x n
  long long* Pb = As + (size_t)max_rows * n;         // [2][n] p of the next column, by all CTAs
  long long* Xb = Pb + 2 * n;                        // [2][n] the next column
  long long* Xc = Xb + 2 * n;                        // [n] the updated column
  Fx* Ub = (Fx*)(Xc + n);                            // [2][n] reflectors u, u'
  Fx* Wb = Ub + 2 * n;                               // [n]
  __shared__ long long redk[VW], red[2][NWARPS];
  __shared__ int s_small;
  __shared__ unsigned redm[VW];
  __shared__ double cmax[MAX_CL], cfro[MAX_CL];
  __shared__ Scal scb[2];                          // by column parity

  // ---- ||A||_inf and ||A||_F^2: a warp per own row, lanes along the row (the lower triangle is
  // referenced) ----
  if (warp < NWARPS) {
    double m = 0.0, f = 0.0;
    for (int lr = warp; lr < rows; lr += NWARPS) {
      const int r = lr * CL + rank;
      double s = 0.0;
#pragma unroll 4
      for (int c = lane; c < n; c += 32) {
        const double x = c <= r ? a.A[r + a.lda * c] : a.A[c + a.lda * r];
        s += fabs(x);
        f = fma(x, x, f);
      }
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      m = s > m || s != s ? s : m;                   // (a NaN stays: comparisons with it fail)
    }
    for (int o = 16; o > 0; o >>= 1) f += __shfl_xor_sync(0xffffffffu, f, o);
    if (lane == 0) {
      ((double*)red[0])[warp] = m;
      ((double*)red[1])[warp] = f;
    }
  }
  __syncthreads();
  if (tid < CL) {
    double m = 0.0, f = 0.0;
    for (int w = 0; w < NWARPS; ++w) {
      const double s = ((double*)red[0])[w];
      m = s > m || s != s ? s : m;
      f += ((double*)red[1])[w];
    }
    *cl.map_shared_rank(&cmax[rank], tid) = m;
    *cl.map_shared_rank(&cfro[rank], tid) = f;
  }
  cl.sync();
  double nrm = 0.0, fro = 0.0;
  for (int b = 0; b < CL; ++b) {
    nrm = cmax[b] > nrm || cmax[b] != cmax[b] ? cmax[b] : nrm;
    fro += cfro[b];
  }
  if (!(nrm <= 1.7976931348623157e308)) {            // NaN or infinity: everything NaN
    const double qnan = __longlong_as_double(0x7FF8000000000000ll);
    for (int i = tid; i < n; i += THREADS) {
      if (rank == 0) {
        a.d[i] = qnan;
        a.e[i] = qnan;
        a.tau[i] = qnan;
      }
    }
    for (int j = rank; j < n - 1; j += CL)
      for (int i = j + 1 + tid; i < n; i += THREADS) a.V[i + a.ldv * j] = qnan;
    return;
  }
  // the sum of squares may over- or underflow: it counts only where it is a comfortable number
  if (fro > 1e-200 && fro < 1e300) nrm = fmin(nrm, 1.000001 * sqrt(fro));
  const int E = nrm > 0.0 ? ilogb(nrm) + 1 : 0;      // nrm < 2^E
  // ---- own rows and the first column into fixed point ----
  for (int lr = 0; lr < rows; ++lr) {
    const int r = lr * CL + rank;
    for (int c = tid; c < n; c += THREADS)
      As[(size_t)lr * n + c] = fx_from_double(c <= r ? a.A[r + a.lda * c] : a.A[c + a.lda * r], E);
  }
  for (int i = tid; i < n; i += THREADS) {
    Xb[i] = fx_from_double(a.A[i], E);
    Pb[i] = 0;
    Ub[i] = Fx{0, 0};
    Wb[i] = Fx{0, 0};
  }
  cl.sync();

  int lr0 = rank == 0 ? 1 : 0;                       // own rows beyond column j start here
  for (int j = 0; j < n; ++j) {
    const int par = j & 1;
    const long long* P = Pb + par * n;
    const long long* X = Xb + par * n;
    const Fx* U = Ub + par * n;
    Fx* Un = Ub + (par ^ 1) * n;
    Scal& sc = scb[par];
    if (tid < VT) {
      // ---- K = u^T p ----
      long long Ksum = 0;
      if (j > 0) {
#pragma unroll 1
        for (int i = j + tid; i < n; i += VT) Ksum += fx_mul(fx_split(P[i]), U[i]);
        Ksum = warp_sum64(Ksum);
        if (lane == 0) redk[warp] = Ksum;
        vec_bar();
        Ksum = sum_parts(redk);
      }
      const Fx K = fx_split(Ksum);
      // ---- w and the updated column x; sums of h^2 and of h l' / 4 + l'^2 / 2^35 ----
      const Fx uj = U[j];
      const Fx wj = fx_split(P[j] - fx_mul(K, uj) + 1);
      long long s0 = 0, s1 = 0;
#pragma unroll 1
      for (int i = j + tid; i < n; i += VT) {
        const Fx u = U[i];
        const Fx w = fx_split(P[i] - fx_mul(K, u) + 1);
        const long long x = X[i] - fx_mul2(u, wj, w, uj);
        Wb[i] = w;
        Xc[i] = x;
        if (i > j) {
          const int lo = (int)(unsigned)x, h = (int)(x >> 32) + (int)((unsigned)lo >> 31);
          s0 += wide(h, h);
          s1 += wide(h, lo >> 2) + (wide(lo, lo) >> 35);
        }
      }
      s0 = warp_sum64(s0);
      s1 = warp_sum64(s1);
      if (lane == 0) {
        red[0][warp] = s0;
        red[1][warp] = s1;
      }
      vec_bar();
      int xs = 0;
      for (;;) {
        if (warp == 0) {
          // ---- the reflector's scalars (one warp; all lanes the same values) ----
          s0 = sum_parts(red[0]);
          s1 = sum_parts(red[1]);
          // |x|^2 = s0 2^-60 + s1 2^-89; below 2^-22 the sums have too few bits: x << xs instead
          const bool small = xs == 0 && s0 + (s1 >> 29) < (1ll << 38);
          if (!small) reflector(s0, s1, 2, xs, j >= n - 2, Xc[j], j + 1 < n ? Xc[j + 1] : 0, lane, sc);
          if (lane == 0) s_small = small;
        }
        vec_bar();
        if (!s_small) break;
        unsigned long long mx = 0;            // leading bits of max |x|
#pragma unroll 1
        for (int i = j + 1 + tid; i < n; i += VT) {
          const long long x = Xc[i];
          const unsigned long long ax = (unsigned long long)(x < 0 ? -x : x);
          mx = mx > ax ? mx : ax;
        }
        unsigned m = mx ? 64u - (unsigned)__clzll((long long)mx) : 0u;
        m = __reduce_max_sync(0xffffffffu, m);
        if (lane == 0) redm[warp] = m;
        vec_bar();
        m = __reduce_max_sync(0xffffffffu, lane < VW ? redm[lane] : 0u);
        xs = m ? 55 - (int)m : -1;            // max |x| << xs in [2^54, 2^55); -1: x = 0
        s0 = s1 = 0;
        if (xs > 0)
#pragma unroll 1
          for (int i = j + 1 + tid; i < n; i += VT) {
            const long long x = Xc[i] << xs;
            const int lo = (int)(unsigned)x, h = (int)(x >> 32) + (int)((unsigned)lo >> 31);
            s0 += wide(h, h);
            s1 += wide(h, lo >> 2) + (wide(lo, lo) >> 35);
          }
        s0 = warp_sum64(s0);
        s1 = warp_sum64(s1);
        if (lane == 0) {
          red[0][warp] = s0;
          red[1][warp] = s1;
        }
        vec_bar();
      }
      // ---- u' ----
      {
        const Fx f = fx_split(sc.f);
        const int sh = sc.sh;
        const bool zero = sc.zero != 0;
#pragma unroll 1
        for (int i = j + 1 + tid; i < n; i += VT) {
          long long u = 0;
          if (!zero) u = i == j + 1 ? sc.u1 : fx_mul(fx_split(Xc[i] << sh), f);
          Un[i] = fx_split(u + 1);                  // (the split keeps 61 bits: to nearest)
        }
      }
    }
    __syncthreads();
    if (warp < NWARPS) {
      // ---- big pass over the own rows r > j, two rows of a warp at a time ----
      int lr = warp + lr0;
      for (; lr + NWARPS < rows; lr += 2 * NWARPS)
        row_pass<2>(As, lr, n, j, CL, rank, par, lane, U, Wb, Un, Pb, Xb, cl);
      if (lr < rows) row_pass<1>(As, lr, n, j, CL, rank, par, lane, U, Wb, Un, Pb, Xb, cl);
      // (the first own row beyond column j + 1)
      if (lr0 * CL + rank <= j + 1) ++lr0;
    } else {
      // ---- output warp: it arrives first and writes while the others go on; what it reads stays
      // until the second column from here ----
      cl.barrier_arrive();
      const Scal& t = scb[par];
      if (rank == 0 && lane < 3) {
        // lane 0: d, lane 1: e, lane 2: tau
        long long v = t.dj;
        int k = E + 1 - 62;
        double* out = a.d + j;
        if (lane == 1) {
          v = t.zero ? t.alpha : (t.neg ? t.nx : -t.nx);
          if (!t.zero) k -= t.sh;
          out = a.e + j;
        } else if (lane == 2) {
          const Fx u1 = fx_split(t.u1);
          v = fx_mul(u1, u1);
          k = 1 - 62;
          out = a.tau + j;
        }
        const double x = fx_to_double(v, k);
        if (lane == 0 || j < n - 1) *out = x;
      }
      if (j < n - 1) {
        // v = u / u1 (unit first entry): u 2 g, with the sign of u1
        const Fx g = fx_split(t.u1 < 0 ? -t.g : t.g);
#pragma unroll 1
        for (int i = j + 1 + 32 * rank + lane; i < n; i += 32 * CL)
          a.V[i + a.ldv * j] = i == j + 1 ? 1.0 : fx_to_double(fx_mul(Un[i], g), 1 - 62);
      }
    }
    if (warp < NWARPS) cl.barrier_arrive();
    cl.barrier_wait();
  }
}

// ---------------------------------------------------------------------------------------------
// The same reduction for larger matrices: the whole grid (or a group of CTAs per matrix) works on
// the lower triangle in global memory (L2), converted in place, with one grid barrier per column.
//
// The trailing triangle is cut into tiles of 32 rows x 8 columns; a warp takes a contiguous run of
// tiles, lane = row.  It updates A(i, c), adds y u'_c to its row's sum, parks y in shared memory,
// and the lanes then sum the tile's columns (4 lanes per column, 8 rows each) against u'_i.  Every
// tile's sums are rounded to 64 bits on their own and added to p by integer atomics, so p does not
// depend on the number of CTAs, the runs or the order.  An element costs ~65 instructions (16 wide
// multiply-adds), half of what the row-wise form of the cluster kernel takes per symmetric pair, and
// half its L2 traffic, which is why the triangle is kept here.  The O(n) vector work is repeated by
// every CTA (the same bits), as in k_sytrd.  What only the host reads (d, e, tau, V) is written
// between the arrival at the barrier and the wait.
// Measured, eigenvalues alone, k_sytrd -> this kernel: n = 700 9.9 -> 4.7 ms, 1575 25.7 -> 12.7, 3600
// 109.7 -> 55.7.  Cycles of a column at n = 700 / 1296 / 3600: loads of p and x with the products for K
// 1.4k / 1.7k / 2.5k (an L2 latency and more), K's block sum 0.8k, w and x 0.6k / 0.9k / 1.9k, the
// reflector with the norm's block sum 1.7k, u' 0.3k / 0.4k / 0.9k, the triangle 1.6k / 2.9k / 14.6k (two
// thirds of its time instructions issue), the barrier with the CTAs' differences 4.2k / 4.2k / 5.8k.
// Each of these was worth its 3 to 8 %: the matrix's addresses stepped by lda instead of formed by
// 64-bit products, the tile parked in split form, u and w read as one 16-byte word, no load after the
// barrier's last poll, p_j from shared memory.  Tried and not kept: the tiles through a ring of
// asynchronous copies instead of one tile ahead in registers (the triangle 16k -> 19k cycles), two or
// four vector elements of a thread together (1 to 4 % slower).
// ---------------------------------------------------------------------------------------------
constexpr int GT = 512, GW = GT / 32;     // threads, warps
constexpr int TC = 8, TLD = 33;           // tile columns, padded rows of a warp's shared tile
constexpr int G_SMEM_MAX = 226 * 1024;

__device__ __forceinline__ void grid_parts_sum(long long v, long long* red, long long& out) {
  v = warp_sum64(v);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  long long t = 0;
#pragma unroll
  for (int w = 0; w < GW; ++w) t += red[w];
  out = t;
}

// the last reflector's and w's element of a column, read as one 16-byte word
struct alignas(16) FxPair {
  Fx u, w;
};

// 8 columns of one tile (col: this row of the first): update, row sums, transposed sums.  EDGE: the
// tile meets the diagonal or the last row.
template <bool EDGE>
__device__ __forceinline__ void fx_tile(const long long (&x)[TC], long long* col, long long lda, int i,
                                        int c0, int n, bool rowok, FxPair r,
                                        const FxPair* __restrict__ UW, const Fx* __restrict__ Un,
                                        Fx* tile, int lane, int row0, long long& racc,
                                        long long* pnext) {
  long long hh = 0, cr = 0;
#pragma unroll
  for (int q = 0; q < TC; ++q) {
    const int c = c0 + q;
    const bool ok = !EDGE || (rowok && c <= i);
    const Fx v = Un[EDGE ? min(c, n - 1) : c];
    const FxPair k = UW[EDGE ? min(c, n - 1) : c];
    long long y = x[q] - fx_mul2x(r.u, k.w, r.w, k.u);
    if (ok) __stcg(col, y);
    col += lda;
    if (EDGE && !ok) y = 0;
    const Fx ys = fx_split(y);
    hh += wide(ys.h, v.h);
    cr += wide(ys.h, v.l) + wide(ys.l, v.h) + ll_term(ys.l, v.l);
    tile[q * TLD + lane] = EDGE && c >= i ? Fx{0, 0} : ys;      // strictly lower
  }
  racc += (hh << 2) + ((cr + CR_HALF) >> 29);
  __syncwarp();
  // column q of the tile: lanes q, q + 8, q + 16, q + 24 sum 8 rows each
  const int q = lane & (TC - 1), r8 = (lane >> 3) * 8;
  const Fx* tp = tile + q * TLD + r8;
  hh = cr = 0;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const Fx v = Un[EDGE ? min(row0 + r8 + k, n - 1) : row0 + r8 + k];
    const Fx ys = tp[k];
    hh += wide(ys.h, v.h);
    cr += wide(ys.h, v.l) + wide(ys.l, v.h) + ll_term(ys.l, v.l);
  }
  long long t = (hh << 2) + ((cr + CR_HALF) >> 29);
  t += __shfl_xor_sync(0xffffffffu, t, 8);
  t += __shfl_xor_sync(0xffffffffu, t, 16);
  if (lane < TC && (!EDGE || c0 + q < n))
    atomicAdd((unsigned long long*)(pnext + c0 + q), (unsigned long long)t);
  __syncwarp();
}

struct GridWhole {
  __device__ __forceinline__ int size() const { return (int)gridDim.x; }
  __device__ __forceinline__ int rank() const { return (int)blockIdx.x; }
};
struct GridSlice {
  const int* s;
  __device__ __forceinline__ int size() const { return *(const volatile int*)s; }
  __device__ __forceinline__ int rank() const { return *(const volatile int*)(s + 1); }
};

template <class Grp>
__device__ __forceinline__ void tri_fx_grid_body(const qk_tri_fx_grid_args& a, const Grp grp) {
  extern __shared__ long long sm[];
  __shared__ long long redk[GW], red0[GW], red1[GW];
  __shared__ unsigned redm[GW];
  __shared__ int s_small;
  __shared__ long long s_pj;             // p_j and u_j of the column at hand
  __shared__ Fx s_uj;
  __shared__ double s_dred[GW];
  __shared__ Scal sc;
  const int n = a.n, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int G = grp.size(), rank = grp.rank();
  const int gthread = rank * GT + tid, totthreads = G * GT;
  unsigned epoch = 0;
  FxPair* UW = (FxPair*)sm;              // [n] u of the last reflector and w (p, until w is known)
  Fx* Un = (Fx*)(UW + n);                // [n] u'
  long long* Xc = (long long*)Un;        // x, until u' takes its place element by element
  Fx* tile = Un + n + (size_t)warp * (TC * TLD);
  long long* Ai = (long long*)a.A;
  double* rs = a.work + 3 * (size_t)n;   // row sums of |A| and A^2 (before the loop only)
  double* fs = rs + n;
  long long* pb = (long long*)a.work;    // [3][n] rotating p

  // ---- norms: a warp per row (fixed order within a row; then every CTA adds the rows alike) ----
  for (int r = rank * GW + warp; r < n; r += G * GW) {
    double s = 0.0, f = 0.0;
#pragma unroll 4
    for (int c = lane; c < n; c += 32) {
      const double x = __ldcg(c <= r ? a.A + r + a.lda * c : a.A + c + a.lda * r);
      s += fabs(x);
      f = fma(x, x, f);
    }
    for (int o = 16; o > 0; o >>= 1) {
      s += __shfl_xor_sync(0xffffffffu, s, o);
      f += __shfl_xor_sync(0xffffffffu, f, o);
    }
    if (lane == 0) {
      __stcg(rs + r, s);
      __stcg(fs + r, f);
    }
  }
  if (!qk_grid_barrier(a.bar, G, epoch, a.status)) return;
  double m = 0.0, f = 0.0;
  for (int r = tid; r < n; r += GT) {
    const double s = __ldcg(rs + r);
    m = s > m || s != s ? s : m;
    f += __ldcg(fs + r);
  }
  for (int o = 16; o > 0; o >>= 1) {
    const double s = __shfl_xor_sync(0xffffffffu, m, o);
    m = s > m || s != s ? s : m;
    f += __shfl_xor_sync(0xffffffffu, f, o);
  }
  if (lane == 0) {
    s_dred[warp] = m;
    ((double*)red0)[warp] = f;
  }
  __syncthreads();
  m = f = 0.0;
  for (int w = 0; w < GW; ++w) {
    const double s = s_dred[w];
    m = s > m || s != s ? s : m;
    f += ((double*)red0)[w];
  }
  if (!(m <= 1.7976931348623157e308)) {              // NaN or infinity: everything NaN
    const double qnan = __longlong_as_double(0x7FF8000000000000ll);
    for (int i = gthread; i < n; i += totthreads) a.d[i] = a.e[i] = a.tau[i] = qnan;
    for (int j = rank; j < n - 1; j += G)
#pragma unroll 1
      for (int i = j + 1 + tid; i < n; i += GT) a.V[i + a.ldv * j] = qnan;
    return;
  }
  if (f > 1e-200 && f < 1e300) m = fmin(m, 1.000001 * sqrt(f));
  const int E = m > 0.0 ? ilogb(m) + 1 : 0;
  // ---- the lower triangle into fixed point, in place; p of the first columns zero ----
  for (int c = rank; c < n; c += G)
    for (int i = c + tid; i < n; i += GT)
      __stcg(Ai + i + a.lda * c, fx_from_double(__ldcg(a.A + i + a.lda * c), E));
  for (int i = gthread; i < 3 * n; i += totthreads) __stcg(pb + i, 0ll);
  for (int i = tid; i < n; i += GT) Un[i] = Fx{0, 0};  // the first column has no update: u = p = 0
  if (tid == 0) s_uj = Fx{0, 0};
  if (!qk_grid_barrier(a.bar, G, epoch, a.status)) return;

  for (int j = 0; j < n; ++j) {
    // p of this column in pb[j % 3]; the big pass adds into (j + 1) % 3; (j + 2) % 3 is zeroed
    const long long* p = pb + (size_t)(j % 3) * n;
    long long* pnext = pb + (size_t)((j + 1) % 3) * n;
    long long* pz = pb + (size_t)((j + 2) % 3) * n;
#pragma unroll 1
    for (int i = gthread; i < n; i += totthreads) __stcg(pz + i, 0ll);
    // ---- vector work (every CTA) ----
    long long Ks = 0;
    for (int t0 = j + tid; t0 < n; t0 += 4 * GT) {
      long long pv[4], xv[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int i = t0 + q * GT;
        if (i < n) {
          pv[q] = __ldcg(p + i);
          xv[q] = __ldcg(Ai + i + a.lda * j);
        }
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int i = t0 + q * GT;
        if (i < n) {
          const Fx u = Un[i];
          Xc[i] = xv[q];
          UW[i] = FxPair{u, Fx{(int)(unsigned)pv[q], (int)(pv[q] >> 32)}};
          if (i == j) s_pj = pv[q];
          Ks += fx_mul(fx_split(pv[q]), u);
        }
      }
    }
    grid_parts_sum(Ks, redk, Ks);
    const Fx K = fx_split(Ks), uj = s_uj;
    const Fx wj = fx_split(s_pj - fx_mul(K, uj) + 1);
    long long s0 = 0, s1 = 0;
#pragma unroll 1
    for (int i = j + tid; i < n; i += GT) {
      const FxPair k = UW[i];
      const long long pi = (long long)(((unsigned long long)(unsigned)k.w.l << 32) | (unsigned)k.w.h);
      const Fx w = fx_split(pi - fx_mul(K, k.u) + 1);
      const long long x = Xc[i] - fx_mul2(k.u, wj, w, uj);
      UW[i].w = w;
      Xc[i] = x;
      if (i > j) {
        const int lo = (int)(unsigned)x, h = (int)(x >> 32) + (int)((unsigned)lo >> 31);
        s0 += wide(h, h);
        s1 += wide(h, lo >> a.sq) + (wide(lo, lo) >> (33 + a.sq));
      }
    }
    s0 = warp_sum64(s0);
    s1 = warp_sum64(s1);
    if (lane == 0) {
      red0[warp] = s0;
      red1[warp] = s1;
    }
    __syncthreads();
    int xs = 0;
    for (;;) {
      if (warp == 0) {
        s0 = s1 = 0;
#pragma unroll
        for (int w = 0; w < GW; ++w) {
          s0 += red0[w];
          s1 += red1[w];
        }
        // |x|^2 = s0 2^-60 + s1 2^(sq - 91); below 2^-18 the sums have too few bits: x << xs
        const bool small = xs == 0 && s0 + (s1 >> (31 - a.sq)) < (1ll << 42);
        if (!small) reflector(s0, s1, a.sq, xs, j >= n - 2, Xc[j], j + 1 < n ? Xc[j + 1] : 0, lane, sc);
        if (lane == 0) s_small = small;
      }
      __syncthreads();
      if (!s_small) break;
      unsigned long long mx = 0;
#pragma unroll 1
      for (int i = j + 1 + tid; i < n; i += GT) {
        const long long x = Xc[i];
        const unsigned long long ax = (unsigned long long)(x < 0 ? -x : x);
        mx = mx > ax ? mx : ax;
      }
      unsigned mb = mx ? 64u - (unsigned)__clzll((long long)mx) : 0u;
      mb = __reduce_max_sync(0xffffffffu, mb);
      if (lane == 0) redm[warp] = mb;
      __syncthreads();
      mb = __reduce_max_sync(0xffffffffu, lane < GW ? redm[lane] : 0u);
      xs = mb ? a.xbits - (int)mb : -1;     // max |x| << xs below 2^xbits
      s0 = s1 = 0;
      if (xs > 0)
#pragma unroll 1
        for (int i = j + 1 + tid; i < n; i += GT) {
          const long long x = Xc[i] << xs;
          const int lo = (int)(unsigned)x, h = (int)(x >> 32) + (int)((unsigned)lo >> 31);
          s0 += wide(h, h);
          s1 += wide(h, lo >> a.sq) + (wide(lo, lo) >> (33 + a.sq));
        }
      s0 = warp_sum64(s0);
      s1 = warp_sum64(s1);
      if (lane == 0) {
        red0[warp] = s0;
        red1[warp] = s1;
      }
      __syncthreads();
    }
    const Scal t = sc;
    {
      const Fx fx = fx_split(t.f);
#pragma unroll 1
      for (int i = j + 1 + tid; i < n; i += GT) {
        long long u = fx_mul(fx_split(Xc[i] << t.sh), fx);
        if (i == j + 1) u = t.u1;
        if (t.zero) u = 0;
        const Fx us = fx_split(u + 1);
        Un[i] = us;
        if (i == j + 1) s_uj = us;
      }
    }
    __syncthreads();
    // ---- big pass: rows and columns beyond j ----
    const int r0 = j + 1, mm = n - r0;
    if (mm > 0) {
      const int nb = (mm + 31) >> 5;
      const int items = 2 * nb * (nb + 1);             // row block b holds tiles 0 .. 4 b + 3
      const int totwarps = G * GW;
      const int per = (items + totwarps - 1) / totwarps;
      const int it0 = (warp * G + rank) * per, it1 = min(it0 + per, items);
      if (it0 < it1) {
        int bi = (int)((sqrtf(2.0f * (float)it0 + 1.0f) - 1.0f) * 0.5f);
        while (bi > 0 && 2 * bi * (bi + 1) > it0) --bi;
        while (2 * (bi + 1) * (bi + 2) <= it0) ++bi;
        int off = 2 * bi * (bi + 1);
        int i = r0 + 32 * bi + lane;
        bool rowok = i < n;
        FxPair row = UW[min(i, n - 1)];
        long long racc = 0;
        long long x[TC], xn[TC];
        auto edge_of = [&](int b, int c) { return c + TC > r0 + 32 * b || r0 + 32 * b + 32 > n; };
        auto load = [&](long long (&dst)[TC], int ri, bool rok, int b, int c0) {
          const long long* col = Ai + ri + a.lda * c0;
          if (!edge_of(b, c0)) {
#pragma unroll
            for (int q = 0; q < TC; ++q, col += a.lda) dst[q] = __ldcg(col);
          } else {
#pragma unroll
            for (int q = 0; q < TC; ++q, col += a.lda) dst[q] = rok && c0 + q <= ri ? __ldcg(col) : 0;
          }
        };
        load(x, i, rowok, bi, r0 + TC * (it0 - off));
        for (int it = it0; it < it1; ++it) {
          const int c0 = r0 + TC * (it - off);
          // the next tile's loads are in flight while this one is worked on
          int nbi = bi, noff = off;
          if (it + 1 >= off + 4 * bi + 4) {
            noff += 4 * bi + 4;
            ++nbi;
          }
          if (it + 1 < it1) {
            const int ni = r0 + 32 * nbi + lane;
            load(xn, ni, ni < n, nbi, r0 + TC * (it + 1 - noff));
          }
          if (edge_of(bi, c0))
            fx_tile<true>(x, Ai + i + a.lda * c0, a.lda, i, c0, n, rowok, row, UW, Un, tile, lane, r0 + 32 * bi,
                          racc, pnext);
          else
            fx_tile<false>(x, Ai + i + a.lda * c0, a.lda, i, c0, n, rowok, row, UW, Un, tile, lane, r0 + 32 * bi,
                           racc, pnext);
          if (nbi != bi || it + 1 == it1) {
            if (rowok) atomicAdd((unsigned long long*)(pnext + i), (unsigned long long)racc);
            racc = 0;
            bi = nbi;
            off = noff;
            i = r0 + 32 * bi + lane;
            rowok = i < n;
            row = UW[min(i, n - 1)];
          }
#pragma unroll
          for (int q = 0; q < TC; ++q) x[q] = xn[q];
        }
      }
    }
    qk_grid_arrive(a.bar);
    // ---- outputs, while the other CTAs arrive: d, e, tau by one thread, a slice of the V column by
    // one warp of every CTA ----
    if (rank == 0 && tid == 64) {
      a.d[j] = fx_to_double(sc.dj, E + 1 - 62);
      if (j < n - 1) {
        a.e[j] = sc.zero ? fx_to_double(sc.alpha, E + 1 - 62)
                         : fx_to_double(sc.neg ? sc.nx : -sc.nx, E + 1 - 62 - sc.sh);
        const Fx u1 = fx_split(sc.u1);
        a.tau[j] = fx_to_double(fx_mul(u1, u1), 1 - 62);
      }
    }
    if (warp == 1) {
      const Fx g = fx_split(sc.u1 < 0 ? -sc.g : sc.g);
#pragma unroll 1
      for (int i = j + 1 + rank + G * lane; i < n; i += 32 * G)
        a.V[i + a.ldv * j] = i == j + 1 ? 1.0 : fx_to_double(fx_mul(Un[i], g), 1 - 62);
    }
    if (!qk_grid_wait(a.bar, G, epoch, a.status)) return;
  }
}

__global__ void __launch_bounds__(GT, 1) k_tri_fx_grid(qk_tri_fx_grid_args a) {
  tri_fx_grid_body(a, GridWhole{});
}

// request r on its own CTA group (cta0[r] .. cta0[r + 1] - 1)
__global__ void __launch_bounds__(GT, 1)
    k_tri_fx_grid_grouped(const __grid_constant__ qk_tri_fx_grid_group g) {
  __shared__ int s_grp[2];
  int r = 0;
  while (r + 1 < g.nreq && (int)blockIdx.x >= g.cta0[r + 1]) ++r;
  if ((int)blockIdx.x >= g.cta0[g.nreq]) return;
  if (threadIdx.x == 0) {
    s_grp[0] = g.cta0[r + 1] - g.cta0[r];
    s_grp[1] = (int)blockIdx.x - g.cta0[r];
  }
  __syncthreads();
  tri_fx_grid_body(g.req[r], GridSlice{s_grp});
}

size_t fx_grid_smem(int n) { return (size_t)n * 24 + (size_t)GW * TC * TLD * 8; }

size_t fx_smem(int n, int cl) {
  const size_t rows = (n + cl - 1) / cl;
  return rows * n * 8 + (size_t)n * 8 * (2 + 2 + 1 + 2 + 1);
}

}  // namespace

// CTAs of the cluster for a matrix of order n (0: does not fit; 615 is the largest that does).  More
// CTAs shorten the row pass and lengthen the broadcast; a single CTA needs no remote stores.
int qk_tri_fx_cluster(int n) {
  if (n < 2) return 0;
  int cl = n <= 64 ? 1 : n <= 128 ? 4 : n <= 256 ? 8 : 16;
  while (cl < MAX_CL && fx_smem(n, cl) > (size_t)SMEM_MAX) cl *= 2;
  return fx_smem(n, cl) <= (size_t)SMEM_MAX ? cl : 0;
}

// One launch over R matrices, a cluster each (all of the size the largest needs; the result does not
// depend on it).
int qk_tri_fx(qk_ctx* ctx, cudaStream_t stream, int R, const qk_tri_fx_args* req) {
  if (R < 1 || R > QK_TRI_FX_GROUP) return qk_fail(ctx, QK_ERR_ARG, "qk_tri_fx: %d matrices", R);
  static std::once_flag once;
  static cudaError_t attr_err = cudaSuccess;
  std::call_once(once, [] {
    attr_err = cudaFuncSetAttribute(k_tri_fx, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_MAX);
    if (attr_err == cudaSuccess)
      attr_err = cudaFuncSetAttribute(k_tri_fx, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  });
  QK_CK(attr_err);
  FxGroup g;
  int cl = 1;
  for (int r = 0; r < R; ++r) {
    const int c = qk_tri_fx_cluster(req[r].n);
    if (!c) return qk_fail(ctx, QK_ERR_ARG, "qk_tri_fx: n=%d does not fit", req[r].n);
    cl = c > cl ? c : cl;
    g.req[r] = req[r];
  }
  size_t smem = 0;
  for (int r = 0; r < R; ++r) {
    const size_t s = fx_smem(req[r].n, cl);
    smem = s > smem ? s : smem;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(cl * R);
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = cl;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  QK_CK(cudaLaunchKernelEx(&cfg, k_tri_fx, g));
  ctx->launches++;
  return QK_OK;
}

int qk_tri_fx_grid_fits(int n) { return n >= 2 && fx_grid_smem(n) <= (size_t)G_SMEM_MAX; }

namespace {
int fx_grid_attr() {
  static std::once_flag once;
  static cudaError_t attr_err = cudaSuccess;
  std::call_once(once, [] {
    attr_err = cudaFuncSetAttribute(k_tri_fx_grid, cudaFuncAttributeMaxDynamicSharedMemorySize, G_SMEM_MAX);
    if (attr_err == cudaSuccess)
      attr_err = cudaFuncSetAttribute(k_tri_fx_grid_grouped, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      G_SMEM_MAX);
  });
  return (int)attr_err;
}
// the sums of h l' / 2^sq stay below 2^63 (|x| < 1/2): sqrt(n) 2^29 2^(31 - sq) < 2^63
int fx_sq(int n) {
  int sq = 2;
  while ((1ll << (2 * (sq + 3))) < (long long)n * 4 + 4) ++sq;
  return sq;
}
// 2^xbits sqrt(n) <= 2^61: a vector of elements below 2^xbits has a norm below 1/2
int fx_xbits(int n) {
  int b = 61;
  for (long long s = 1; s < n; s *= 4) --b;
  return b;
}
}  // namespace

// cooperative launch over `grid` CTAs (one per SM)
int qk_tri_fx_grid(qk_ctx* ctx, int grid, qk_tri_fx_grid_args a) {
  QK_CK((cudaError_t)fx_grid_attr());
  a.sq = fx_sq(a.n);
  a.xbits = fx_xbits(a.n);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(GT);
  cfg.dynamicSmemBytes = fx_grid_smem(a.n);
  cfg.stream = ctx->stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  QK_CK(cudaLaunchKernelEx(&cfg, k_tri_fx_grid, a));
  ctx->launches++;
  return QK_OK;
}

int qk_tri_fx_grid_launch_group(qk_ctx* ctx, cudaStream_t stream, qk_tri_fx_grid_group& g) {
  QK_CK((cudaError_t)fx_grid_attr());
  size_t smem = 0;
  for (int r = 0; r < g.nreq; ++r) {
    g.req[r].sq = fx_sq(g.req[r].n);
    g.req[r].xbits = fx_xbits(g.req[r].n);
    const size_t s = fx_grid_smem(g.req[r].n);
    smem = s > smem ? s : smem;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(g.cta0[g.nreq]);
  cfg.blockDim = dim3(GT);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  QK_CK(cudaLaunchKernelEx(&cfg, k_tri_fx_grid_grouped, g));
  ctx->launches++;
  return QK_OK;
}

// k_gemm_tc.cu -- FP64 GEMM by exact integer slices on the 5th-generation tensor cores.
//
// C_b = alpha op(A_b) op(B_b) + beta C_b (FP64, column-major, strided batch), the contract of
// qk_dgemm.  GB300 issues one FP64 warp instruction per 64 cycles and SM sub-partition (about
// 1.2 TFLOP/s), so the DFMA kernel is bound by that pipe whatever its tiling; the BF16 tensor
// pipe is ~1600 times faster.  The product is therefore formed from integers that BF16 operands
// and FP32 accumulators hold exactly (the error-free splitting of Ozaki, Ogita, Oishi and Rump,
// "Error-free transformations of matrix multiplication by using fast routines of matrix
// multiplication and its applications", Numer. Algorithms 59, 2012):
//
//   row i of op(A), max |a_ik| < 2^(E_i):  a_ik = 2^(E_i - 62) q_ik,  q_ik an integer, |q| < 2^62
//   (exact for |a_ik| >= 2^-10 of the row's power of two, else rounded to 2^(E_i - 62)), and
//   q = sum_s d_s 256^(7-s) with eight balanced digits, -128 <= d_s <= 127; columns of op(B)
//   likewise.  Digits are exact in BF16, a digit product is an integer of at most 2^14, and
//   G_g = sum_k sum_(s+t=g) d_s(a) d_t(b), g = 0..7 (36 digit products), is an integer below
//   8 * 128 * 2^14 = 2^24 over 128 k: exact in the FP32 accumulators of tensor memory.
//
// After every 128 k the epilogue adds the eight G_g into a 112-bit integer per element (two
// 64-bit halves); one rounding to FP64 ends the sum.  What is left out (g >= 8) and rounded is
// below K 2^-60 of max_k |a_ik| max_k |b_kj|, against K 2^-53 of sum_k |a b| for the DFMA chain:
// over the framework's contractions the result is closer to the exact product than DFMA's.
// (An operand whose k scales differ wildly, so that sum |a b| is far below max |a| max |b|, would
// lose that advantage: qk_dgemm_dev, which takes any matrix, and qsGW's Fock algebra stay on DFMA.)
// Where k runs over the caller's basis functions, whose norms are the caller's choice, and op(B) holds
// orbital coefficients (qk_gemm_tc_basis), their scale per k moves to op(A) as a power of two before
// both are sliced: the result then has the same bits whatever powers of two the functions are scaled
// by, as with DFMA.
// The integers make the result independent of the order of summation.
//
// Non-finite operands: a row (column) with a NaN gives NaN; an element whose row or column holds
// an infinity is summed again in FP64 from the operands, so that infinities come out as they do
// from DFMA.
//
// Kernel (persistent, one 128 x 64 output tile at a time per CTA, 640 threads):
//   warp 0 lane 0 : cp.async.bulk of the 8 A and 8 B digit planes of a 32-wide k block into one of
//                   two stages (64 KB + 32 KB; the planes are stored in global memory as the
//                   64-byte-swizzled shared-memory image, so a stage is two plain bulk copies)
//   warp 1        : the 36 digit products of a stage as 12 tcgen05.mma (M=128, K=16) per k-step: A
//                   digit s times several B digits side by side (N = 64 each, up to 256) adds to
//                   the adjacent groups G_g, which lie side by side in TMEM (8 x 64 = all 512
//                   columns).  A is then read from shared memory 12 times instead of 36, and the
//                   kernel is bound by the tensor pipe; one MMA per digit pair (N = 64) took 64
//                   cycles for 32 cycles of tensor work
//   warps 4..19   : drain G_g while the tensor cores work on the later groups, then assemble the
//                   FP64 result while they work on the next tile
// Measured (one GB300, preparation included): 3600 x 3600 x 3600 in 2.30 ms (40.6 TFLOP/s; DFMA
// 78.7 ms, 1.19), 25600 x 2800 x 480 in 1.69 ms (DFMA 55.6), 3600 x 3600 x 128 in 0.10 ms (DFMA
// 2.85).  A 128-k chunk takes ~13.1k cycles of MMA issue against 9.2k at the nominal tensor rate,
// and 13.6k with the epilogue draining beside it.
#include <mutex>
#include "qk_tc.cuh"

namespace {

constexpr int TM = 128, TN = 64, KB = 32, NS = 8;  // tile, k block, digit planes
constexpr int CHUNK = 4;                           // k blocks per exact accumulation (128 k)
constexpr int A_PLANE = TM * KB * 2, B_PLANE = TN * KB * 2;      // 8 KB, 4 KB
constexpr int A_STAGE = NS * A_PLANE, B_STAGE = NS * B_PLANE;    // 64 KB, 32 KB
constexpr int STAGES = 2;
constexpr int STAGE_BYTES = A_STAGE + B_STAGE;
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + 256;
constexpr int EPI = 16, EC = TN / (EPI / 4);         // epilogue warps, columns of each
constexpr int NTHREADS = 128 + 32 * EPI;
// registers per thread after the split (launched with 96: 640 x 96 = 128 x 32 + 512 x 112)
#define TC_REGS_IO "32"
#define TC_REGS_EPI "112"
constexpr uint32_t TMEM_COLS = 512;
// D=F32, A=B=BF16, both K-major, M=128 (N is added per MMA)
constexpr uint32_t IDESC0 = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(TM >> 4) << 24);
constexpr unsigned HI_INF = 0x7FF00000u, HI_NAN = 0x7FF80000u;

struct Operand {           // op(A) as rows x K, or op(B)^T as rows x K
  const double* X;         // X(r, k) = X[r + ld k] (trans = 0) or X[k + ld r]
  long long ld, stride;    // stride between batch entries (0: one shared operand)
  int rows, rb, trans;     // rb: rows per plane block (TM for A, TN for B)
  int row_blocks, batch;   // batch: plane sets (1: shared by all batch entries)
  const double* kscale;    // optional factors of the k index: X(r, k) kscale[k + sk b]
  long long sk;
  const int* kexp;         // optional exponents of the k index (one operand's negated): X(r, k) 2^kexp[k]
  int kneg;
  uint8_t* P;              // digit planes: [batch][row block][k block][digit][rb rows][64 B]
  unsigned* info;          // per row: high word of max |x| (exponent; Inf and NaN codes)
  unsigned* part;          // partial maxima [batch][k slab][row] (slabs > 0)
  int slabs;               // 0: the slicing kernel finds the maxima itself (K <= SELF_K)
};

struct TcGemm {
  Operand a, b;
  int M, N, K, kblks, mt, nt, batch, slices, kb_per_slice, lower;
  double alpha, beta;
  double* C;
  long long ldc, sC;
};

// ---- operand preparation -----------------------------------------------------------------------
// x 2^e (|e| <= KEXP_MAX), on the integer pipe where x and the result are normal numbers
__device__ __forceinline__ double mul_pow2(double x, int e) {
  const int hi = __double2hiint(x), lo = __double2loint(x), ex = (hi >> 20) & 0x7FF;
  if (ex != 0 && ex != 0x7FF && (unsigned)(ex + e - 1) < 2046u) return __hiloint2double(hi + (e << 20), lo);
  return ((hi & 0x7FFFFFFF) | lo) ? x * __hiloint2double((e + 1023) << 20, 0) : x;
}
__device__ __forceinline__ double at_k(const Operand& o, const double* ks, double x, int k) {
  if (o.kexp) return mul_pow2(x, o.kneg ? -__ldg(o.kexp + k) : __ldg(o.kexp + k));
  return ks ? x * ks[k] : x;
}
__device__ __forceinline__ unsigned abs_hi(double x) {
  const unsigned hi = (unsigned)__double2hiint(x) & 0x7FFFFFFFu;
  return (hi >= HI_INF && (hi > HI_INF || __double2loint(x) != 0)) ? HI_NAN : hi;
}

constexpr int SELF_K = 128;
constexpr int KEXP_MAX = 400;

// kexp[k] = exponent of the largest |c(k, j)| (0 where that is zero or not finite), a warp per k.  A launch
// of its own, ~3 us: once per transformation (26 functions 129 us with one per quarter, 117 with one, 120
// without scales; 30: 164, 153, 150; 60: 839, 823, 958).
__global__ void __launch_bounds__(256) k_tc_kexp(Operand b, int K, int* __restrict__ kexp) {
  const int lane = threadIdx.x & 31, k = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (k >= K) return;
  unsigned m = 0;
  for (int r = lane; r < b.rows; r += 32) m = max(m, abs_hi(b.trans ? b.X[k + b.ld * r] : b.X[r + b.ld * k]));
  m = __reduce_max_sync(0xffffffffu, m);
  const int e = (int)(m >> 20) - 1023;
  if (lane == 0) kexp[k] = m == 0u || m >= HI_INF ? 0 : max(-KEXP_MAX, min(KEXP_MAX, e));
}

// part[slab][r] = max over the slab's k of the high word of |X(r, k)|; 256 threads.  trans = 0: 32
// rows x 256 k per block, lanes along the rows; trans = 1: 8 rows x 1024 k, a warp along k.
__global__ void __launch_bounds__(256) k_tc_rowmax(Operand a, Operand b, int K, int a_blocks) {
  __shared__ unsigned red[8][32];
  int bid = blockIdx.x;
  const bool isA = bid < a_blocks;
  if (!isA) bid -= a_blocks;
  const Operand o = isA ? a : b;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int rows_per = o.trans ? 8 : 32, strips = (o.rows + rows_per - 1) / rows_per;
  const int ks = bid % o.slabs;
  bid /= o.slabs;
  const int strip = bid % strips, bt = bid / strips;
  const double* __restrict__ X = o.X + (long long)bt * o.stride;
  const double* sc = o.kscale ? o.kscale + (long long)bt * o.sk : nullptr;
  unsigned* out = o.part + ((size_t)bt * o.slabs + ks) * o.row_blocks * o.rb;
  unsigned m = 0;
  if (o.trans) {
    const int r = strip * 8 + ty;
    if (r < o.rows) {
      const int k1 = min(K, ks * 1024 + 1024);
#pragma unroll 8
      for (int k = ks * 1024 + tx; k < k1; k += 32) m = max(m, abs_hi(at_k(o, sc, X[k + o.ld * r], k)));
    }
    m = __reduce_max_sync(0xffffffffu, m);
    if (tx == 0 && r < o.rows) out[r] = m;
  } else {
    const int r = strip * 32 + tx;
    if (r < o.rows) {
      const int k1 = min(K, ks * 256 + 256);
#pragma unroll 8
      for (int k = ks * 256 + ty; k < k1; k += 8) m = max(m, abs_hi(at_k(o, sc, X[r + o.ld * k], k)));
    }
    red[ty][tx] = m;
    __syncthreads();
    if (ty == 0) {
#pragma unroll
      for (int i = 1; i < 8; ++i) m = max(m, red[i][tx]);
      if (r < o.rows) out[r] = m;
    }
  }
}

// x = 2^(E - 62) q with E - 1 the exponent of the row's maximum; the bytes of the returned word
// are d_s + 128 (byte 7: s = 0), by adding 128 to every byte position at once
__device__ __forceinline__ unsigned long long digits_of(double x, int exmax) {
  const unsigned long long bits = (unsigned long long)__double_as_longlong(x);
  const int ex = (int)((bits >> 52) & 0x7FF);
  const unsigned long long m = (bits & 0xFFFFFFFFFFFFFull) | (ex ? 1ull << 52 : 0ull);
  const int sh = max(ex, 1) - max(exmax, 1) + 9;
  unsigned long long q;
  if (sh >= 0) q = m << sh;
  else if (sh > -63) q = (m + (1ull << (-sh - 1))) >> -sh;
  else q = 0;
  if ((long long)bits < 0) q = 0ull - q;
  return q + 0x8080808080808080ull;
}

// Digit planes of 32 rows per block of 128 threads: the doubles are staged in shared memory, then a
// thread takes 8 consecutive k of one row and writes one 16-byte piece per plane (a warp writes 512
// contiguous bytes).  Memory-bound by design: 8 bytes read, 16 written per element.
// SELF (K <= SELF_K): a block takes all k of its rows and finds their maxima on the way (with a block
// per 32 k and a scan of the rows in each, rows beyond L2's reach were read once more per block: the
// AO to MO transformation of 96 functions, 6.15 -> 5.56 ms; 4.73 since a lane's eight loads along k are
// issued before any of them is scaled).
// Otherwise a block takes 32 k and the maxima come from k_tc_rowmax.
template <bool SELF>
__global__ void __launch_bounds__(128) k_tc_slice(Operand a, Operand b, int K, int kblks,
                                                  int a_blocks) {
  constexpr int KBS = SELF ? SELF_K / KB : 1;            // k blocks of a CTA, at most
  __shared__ double t[KBS][32][33];
  __shared__ unsigned smax[4][32];
  int bid = blockIdx.x;
  const bool isA = bid < a_blocks;
  if (!isA) bid -= a_blocks;
  const Operand o = isA ? a : b;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int strips = o.row_blocks * (o.rb / 32);
  const int strip = bid % strips;
  bid /= strips;
  const int kb0 = SELF ? 0 : bid % kblks, bt = SELF ? bid : bid / kblks;
  const int nkb = SELF ? kblks : 1;
  const int r0 = strip * 32;
  const double* __restrict__ X = o.X + (long long)bt * o.stride;
  const double* sc = o.kscale ? o.kscale + (long long)bt * o.sk : nullptr;
  const size_t rows_pad = (size_t)o.row_blocks * o.rb;
  unsigned m[8] = {};                                    // trans: of rows ty + 4 i; else m[0]: row tx
#pragma unroll
  for (int q = 0; q < KBS; ++q) {
    if (q >= nkb) break;
    const int k0 = (kb0 + q) * KB;
    double v[8];
    if (o.trans) {
      const int k = k0 + tx;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int r = r0 + ty + 4 * i;
        v[i] = (r < o.rows && k < K) ? X[k + o.ld * r] : 0.0;
      }
      if ((sc || o.kexp) && k < K) {
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = at_k(o, sc, v[i], k);
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        t[q][ty + 4 * i][tx] = v[i];
        if (SELF) m[i] = max(m[i], abs_hi(v[i]));
      }
    } else {
      const int r = r0 + tx;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int k = k0 + ty + 4 * i;
        v[i] = (r < o.rows && k < K) ? at_k(o, sc, X[r + o.ld * k], k) : 0.0;
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        t[q][tx][ty + 4 * i] = v[i];
        if (SELF) m[0] = max(m[0], abs_hi(v[i]));
      }
    }
  }
  // the rows' maxima
  if (SELF && o.trans) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const unsigned mr = __reduce_max_sync(0xffffffffu, m[i]);
      if (tx < 4) smax[tx][ty + 4 * i] = mr;
    }
  } else {
    if (!SELF && r0 + tx < o.rows)
      for (int i = ty; i < o.slabs; i += 4)
        m[0] = max(m[0], o.part[((size_t)bt * o.slabs + i) * rows_pad + r0 + tx]);
    smax[ty][tx] = m[0];
  }
  __syncthreads();
  const int rl = threadIdx.x >> 2, c = threadIdx.x & 3;  // row, 16-byte piece (8 k)
  const int r = r0 + rl;
  const unsigned info = max(max(smax[0][rl], smax[1][rl]), max(smax[2][rl], smax[3][rl]));
  if (kb0 == 0 && c == 0) o.info[bt * rows_pad + r] = info;
  const int exmax = (int)(info >> 20);
  const bool ok = info < HI_INF;
  const int rb = r / o.rb, rr = r - rb * o.rb;
  const size_t plane = (size_t)o.rb * 64;
  uint8_t* base = o.P + ((((size_t)bt * o.row_blocks + rb) * kblks + kb0) * NS) * plane +
                  (size_t)rr * 64 + ((c ^ ((rr >> 1) & 3)) << 4);
  for (int q = 0; q < nkb; ++q, base += NS * plane) {
    unsigned long long d[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) d[i] = digits_of(ok ? t[q][rl][c * 8 + i] : 0.0, ok ? exmax : 1);
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      uint32_t w[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        // byte -> float without a conversion instruction: 2^23 + byte, minus 2^23 + 128; the upper
        // half of the float is the BF16 value (digits have at most 8 significant bits)
        const unsigned w0 = s < 4 ? (unsigned)(d[2 * i] >> 32) : (unsigned)d[2 * i];
        const unsigned w1 = s < 4 ? (unsigned)(d[2 * i + 1] >> 32) : (unsigned)d[2 * i + 1];
        const unsigned sel = 0x7650u | (unsigned)(3 - (s & 3));
        const float f0 = __uint_as_float(__byte_perm(w0, 0x4B000000u, sel)) - 8388736.0f;
        const float f1 = __uint_as_float(__byte_perm(w1, 0x4B000000u, sel)) - 8388736.0f;
        w[i] = __byte_perm(__float_as_uint(f0), __float_as_uint(f1), 0x7632u);
      }
      *(uint4*)(base + s * plane) = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
}

// ---- GEMM ----------------------------------------------------------------------------------------
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes,
                                          uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          su32(dst)),
      "l"(src), "r"(bytes), "r"(su32(bar))
      : "memory");
}

__device__ __forceinline__ uint64_t sdesc_sw64(const void* tile) {
  const uint32_t a = su32(tile);
  uint64_t d = 0;
  d |= (uint64_t)((a & 0x3FFFF) >> 4);      // start address
  d |= (uint64_t)1 << 16;                   // leading byte offset (unused for swizzled K-major)
  d |= (uint64_t)(512 >> 4) << 32;          // stride byte offset: 8 rows x 64 B
  d |= (uint64_t)1 << 46;                   // descriptor version (tcgen05)
  d |= (uint64_t)4 << 61;                   // 64-byte swizzle
  return d;
}

__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(p));
  return p != 0;
}

struct Unit {
  int m, n, b, z, kb0, kb1;
};
// unit u of the launch: tiles in groups of 8 row blocks walked along n, so that the CTAs running at
// one time share about as many A rows as B rows in L2
__device__ __forceinline__ Unit unit_of(const TcGemm& g, int u) {
  const int tiles = g.mt * g.nt;
  Unit t;
  const int bz = u / tiles, idx = u - bz * tiles;
  t.b = bz / g.slices;
  t.z = bz - t.b * g.slices;
  const int per = 8 * g.nt, gi = idx / per, first = gi * 8, gsz = min(8, g.mt - first);
  const int r = idx - gi * per;
  t.n = r / gsz;
  t.m = first + r - t.n * gsz;
  t.kb0 = t.z * g.kb_per_slice;
  t.kb1 = min(g.kblks, t.kb0 + g.kb_per_slice);
  return t;
}
__device__ __forceinline__ bool skip_unit(const TcGemm& g, const Unit& t) {
  return g.lower && (t.m + 1) * TM <= t.n * TN;  // strictly above the diagonal
}

// 2^s T of the integer T = hi 2^32 + lo (|T| < 2^95) rounded to nearest even, s = e - 2112 with e
// the sum of the two biased row exponents, on the integer pipe (the FP64 pipe takes 64 cycles per
// warp conversion) and without branches: |T| as three 32-bit words, normalised to 64 bits plus a
// sticky word.  `biased` is the result's exponent; outside the normal range the value returned has
// exponent 1023 and is to be scaled (assemble_scaled).
__device__ __forceinline__ double assemble(long long hi, long long lo, int e, int& biased) {
  unsigned long long L = ((unsigned long long)hi << 32) + (unsigned long long)lo;
  const int top = (int)(hi >> 32) + (int)(lo >> 63) + (L < (unsigned long long)lo ? 1 : 0);
  const int m = top >> 31;
  L = (L ^ (unsigned long long)(long long)m) - (unsigned long long)(long long)m;
  unsigned a = (unsigned)(top ^ m) + (L == 0ull ? (unsigned)-m : 0u);
  unsigned b = (unsigned)(L >> 32), c = (unsigned)L;
  const bool z1 = a == 0u;
  a = z1 ? b : a;
  b = z1 ? c : b;
  c = z1 ? 0u : c;
  const bool z2 = a == 0u;  // (then c is 0)
  a = z2 ? b : a;
  b = z2 ? 0u : b;
  const int z = __clz((int)a) & 31;
  const unsigned A = __funnelshift_l(b, a, z), B = __funnelshift_l(c, b, z), S = c << z;
  // 53 bits of A:B; the discarded 11 bits and the sticky word decide the rounding
  const unsigned mlo = __funnelshift_r(B, A, 11);
  const unsigned rem = ((B & 0x7FFu) << 1) | (S ? 1u : 0u);
  biased = a ? e - z - (z1 ? 32 : 0) - (z2 ? 32 : 0) + (96 - 1 - 2112 + 1023) : 1;
  unsigned long long bits = (((unsigned long long)(A >> 11) << 32) | mlo) +
                            (rem + (mlo & 1u) > 0x800u ? 1ull : 0ull);
  const int bx = (unsigned)(biased - 1) < 2045u ? biased : 1023;
  bits += (unsigned long long)(unsigned)(bx - 1) << 52;
  bits |= (unsigned long long)((unsigned)m & 0x80000000u) << 32;
  return __longlong_as_double((long long)bits);
}
// v 2^(biased - 1023) in FP64 steps (overflow and subnormal results as the format has them)
__device__ __forceinline__ double assemble_scaled(double v, int biased) {
  const int k = max(-2400, min(2400, biased - 1023)), k3 = k / 3, k1 = k - 2 * k3;
  const double f3 = __longlong_as_double((long long)(k3 + 1023) << 52);
  return v * f3 * f3 * __longlong_as_double((long long)(k1 + 1023) << 52);
}

__device__ __noinline__ double plain_dot(const TcGemm& g, const Unit& t, int row, int col) {
  const double* X = g.a.X + (long long)t.b * g.a.stride;
  const double* Y = g.b.X + (long long)t.b * g.b.stride;
  const double* ks = g.b.kscale ? g.b.kscale + (long long)t.b * g.b.sk : nullptr;
  const int k1 = min(g.K, t.kb1 * KB);
  double s = 0.0;
  for (int k = t.kb0 * KB; k < k1; ++k)
    s = fma(at_k(g.a, nullptr, g.a.trans ? X[k + g.a.ld * row] : X[row + g.a.ld * k], k),
            at_k(g.b, ks, g.b.trans ? Y[k + g.b.ld * col] : Y[col + g.b.ld * k], k), s);
  return s;
}

__device__ __forceinline__ void tmem_ld16x2(uint32_t t0, uint32_t t1, uint32_t (&r)[16],
                                            uint32_t (&s)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,"
      "%15}, [%32];\n"
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,"
      "%28,%29,%30,%31}, [%33];\n"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(s[0]), "=r"(s[1]), "=r"(s[2]), "=r"(s[3]), "=r"(s[4]),
        "=r"(s[5]), "=r"(s[6]), "=r"(s[7]), "=r"(s[8]), "=r"(s[9]), "=r"(s[10]), "=r"(s[11]),
        "=r"(s[12]), "=r"(s[13]), "=r"(s[14]), "=r"(s[15])
      : "r"(t0), "r"(t1)
      : "memory");
}

// groups 2 p and 2 p + 1 into one 64-bit half per element, at weights w and w / 256
__device__ __forceinline__ bool drain_pair(uint32_t tq, int p, int w, uint64_t* acc_full,
                                           uint64_t* acc_empty, uint32_t ch, int lane, int* status,
                                           long long (&acc)[EC]) {
  const bool have = mbar_wait(&acc_full[p], ch & 1, status);
  if (!__all_sync(0xffffffffu, have)) return false;
  tc_fence_after();
  uint32_t r[EC], s[EC];
  tmem_ld16x2(tq + (uint32_t)(2 * p * TN), tq + (uint32_t)((2 * p + 1) * TN), r, s);
  tc_fence_before();
  __syncwarp();
  if (lane == 0) mbar_arrive(&acc_empty[p]);
#pragma unroll
  for (int j = 0; j < EC; ++j) {
    acc[j] += (long long)__float2int_rn(__uint_as_float(r[j])) * w;
    acc[j] += (long long)__float2int_rn(__uint_as_float(s[j])) * (w >> 8);
  }
  return true;
}

__global__ void __launch_bounds__(NTHREADS, 1) k_gemm_tc(const __grid_constant__ TcGemm g,
                                                         int* status) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* full = (uint64_t*)(smem + STAGES * STAGE_BYTES);
  uint64_t* empty = full + STAGES;
  uint64_t* acc_full = empty + STAGES;     // [4] pair of groups finished by the tensor cores
  uint64_t* acc_empty = acc_full + NS / 2; // [4] pair drained by the epilogue warps
  uint64_t* drain = acc_empty + NS / 2;
  uint32_t* tmem_slot = (uint32_t*)(drain + 1);
  int* abort_flag = (int*)(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int units = g.mt * g.nt * g.batch * g.slices;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int i = 0; i < NS / 2; ++i) {
      mbar_init(&acc_full[i], 1);
      mbar_init(&acc_empty[i], EPI);  // one arrival per epilogue warp
    }
    mbar_init(drain, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     su32(tmem_slot)),
                 "r"(TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 " TC_REGS_IO ";");
    if (warp == 0) {
      if (lane == 0) {
        // ---------------- producer ----------------
        uint32_t it = 0;
        bool ok = true;
        for (int u = blockIdx.x; u < units && ok; u += gridDim.x) {
          const Unit t = unit_of(g, u);
          if (skip_unit(g, t)) continue;
          const uint8_t* pa =
              g.a.P + ((size_t)((g.a.batch > 1 ? t.b : 0) * (long long)g.a.row_blocks + t.m) * g.kblks) * A_STAGE;
          const uint8_t* pb =
              g.b.P + ((size_t)((g.b.batch > 1 ? t.b : 0) * (long long)g.b.row_blocks + t.n) * g.kblks) * B_STAGE;
          for (int kb = t.kb0; kb < t.kb1; ++kb, ++it) {
            const int s = it % STAGES;
            if (!mbar_wait(&empty[s], ((it / STAGES) & 1) ^ 1, status)) {
              *(volatile int*)abort_flag = 1;
              ok = false;
              break;
            }
            if (*(volatile int*)abort_flag) { ok = false; break; }
            uint8_t* st = smem + s * STAGE_BYTES;
            mbar_expect_tx(&full[s], STAGE_BYTES);
            bulk_load(st, pa + (size_t)kb * A_STAGE, A_STAGE, &full[s]);
            bulk_load(st + A_STAGE, pb + (size_t)kb * B_STAGE, B_STAGE, &full[s]);
          }
        }
        // every issued stage must have landed before the CTA may exit
        for (uint32_t i = (it > STAGES ? it - STAGES : 0); i < it; ++i)
          mbar_wait(&full[i % STAGES], (i / STAGES) & 1, status);
      }
      __syncwarp();
    } else if (warp == 1) {
      // ---------------- MMA issuer ----------------
      // The whole warp walks the loops and one elected lane issues: the descriptors are then
      // warp-uniform values (uniform registers) and the 72 MMAs of a stage are straight-line code.
      const bool leader = elect_one();
      const uint64_t d0 = sdesc_sw64(smem);
      uint32_t it = 0, ch = 0;
      bool ok = true;
      for (int u = blockIdx.x; u < units && ok; u += gridDim.x) {
        const Unit t = unit_of(g, u);
        if (skip_unit(g, t)) continue;
        for (int kc = t.kb0; kc < t.kb1 && ok; kc += CHUNK, ++ch) {
          const int ke = min(t.kb1, kc + CHUNK);
          for (int kb = kc; kb < ke; ++kb, ++it) {
            const int s = it % STAGES;
            ok = mbar_wait(&full[s], (it / STAGES) & 1, status) && !*(volatile int*)abort_flag;
            if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
            tc_fence_after();
            const uint64_t da0 = d0 + (uint64_t)(s * (STAGE_BYTES >> 4));
            const uint64_t db0 = da0 + (uint64_t)(A_STAGE >> 4);
            const bool first = kb == kc, last = kb == ke - 1;
            // A digit i times B digits t0, t0 + 1, .. side by side (their planes are contiguous, so
            // they form one operand of up to 256 rows) lands in the adjacent groups i + t0, ..: first
            // the groups 0..3, then 4..7.  Group i is complete after digit i of its half.
#pragma unroll 1
            for (int h = 0; h < 2; ++h) {
              if (first) {
                for (int pr = 2 * h; pr < 2 * h + 2 && ok; ++pr)
                  ok = mbar_wait(&acc_empty[pr], (ch & 1) ^ 1, status);
                if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
                tc_fence_after();
              }
              if (leader) {
#pragma unroll 1
                for (int i = 0; i < 4 + 4 * h; ++i) {
                  const int g0 = h ? (i > 4 ? i : 4) : i;  // first group, B digit g0 - i
                  const uint64_t da = da0 + (uint64_t)(i * (A_PLANE >> 4));
                  const uint64_t db = db0 + (uint64_t)((g0 - i) * (B_PLANE >> 4));
                  const uint32_t d = tmem + (uint32_t)(g0 * TN);
                  const uint32_t idesc = IDESC0 | ((uint32_t)((4 * h + 4 - g0) * TN >> 3) << 17);
                  umma_bf16(d, da, db, idesc, i > 0 || !first);
                  umma_bf16(d, da + 2, db + 2, idesc, 1);
                  if (last && i >= 4 * h && (i & 1)) umma_commit(&acc_full[i >> 1]);
                }
              }
              __syncwarp();
            }
            if (!ok) break;
            if (leader) umma_commit(&empty[s]);
            __syncwarp();
          }
        }
      }
      if (!ok) {  // let the tensor cores finish before TMEM is freed
        *(volatile int*)abort_flag = 1;
        if (leader) umma_commit(drain);
        __syncwarp();
        mbar_wait(drain, 0, status);
      }
      __syncwarp();
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 " TC_REGS_EPI ";");
    // ---------------- epilogue warps 4..19 ----------------
    const int q = warp & 3;              // TMEM lane quadrant this warp may access
    const int part = (warp - 4) >> 2;    // its 16 of the 64 columns
    const uint32_t tq = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(part * EC);
    uint32_t ch = 0;
    bool ok = true;
    for (int u = blockIdx.x; u < units && ok; u += gridDim.x) {
      const Unit t = unit_of(g, u);
      if (skip_unit(g, t)) continue;
      long long hi[EC], lo[EC];
#pragma unroll
      for (int j = 0; j < EC; ++j) hi[j] = lo[j] = 0;
      for (int kc = t.kb0; kc < t.kb1 && ok; kc += CHUNK, ++ch) {
        // G_g joins its half at weight 256^(3-g) (g < 4) or 256^(7-g)
        ok = drain_pair(tq, 0, 1 << 24, acc_full, acc_empty, ch, lane, status, hi) &&
             drain_pair(tq, 1, 1 << 8, acc_full, acc_empty, ch, lane, status, hi) &&
             drain_pair(tq, 2, 1 << 24, acc_full, acc_empty, ch, lane, status, lo) &&
             drain_pair(tq, 3, 1 << 8, acc_full, acc_empty, ch, lane, status, lo);
        ok = __all_sync(0xffffffffu, ok && !*(volatile int*)abort_flag);
      }
      if (!ok) break;
      const int row = t.m * TM + q * 32 + lane;
      const int c0 = t.n * TN + part * EC;
      const int ba = g.a.batch > 1 ? t.b : 0, bb = g.b.batch > 1 ? t.b : 0;
      const unsigned ia = row < g.M ? g.a.info[(long long)ba * g.a.row_blocks * TM + row] : 0u;
      const unsigned ic = lane < EC && c0 + lane < g.N ? g.b.info[(long long)bb * g.b.row_blocks * TN + c0 + lane] : 0u;
      double* __restrict__ C = g.C + (long long)(t.b * g.slices + t.z) * g.sC + row;
      const bool inrow = row < g.M;
      const int ea = max((int)(ia >> 20), 1);
      const unsigned special = __ballot_sync(0xffffffffu, ic >= HI_INF);
      const bool row_special = ia >= HI_INF;
      // eight columns at a time from the front of hi/lo, then the rest moves up (a rolled loop over
      // register arrays)
#pragma unroll 1
      for (int j0 = 0; j0 < EC; j0 += 8) {
#pragma unroll
        for (int h = 0; h < 8; h += 4) {
          const int col = c0 + j0 + h;
          double* cp = C + g.ldc * col;
          double v[4], cv[4];
          // columns of this group to write: inside C, finite operands
          unsigned wr = col < g.N ? (g.N - col >= 4 ? 0xFu : (1u << (g.N - col)) - 1u) : 0u;
          wr &= ~(special >> (j0 + h));
          if (!inrow || row_special) wr = 0u;
          if (g.beta != 0.0) {
#pragma unroll
            for (int j = 0; j < 4; ++j) cv[j] = (wr >> j) & 1u ? cp[g.ldc * j] : 0.0;
          }
          bool scaled = false;
          int be[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            v[j] = assemble(hi[h + j], lo[h + j],
                            ea + max((int)(__shfl_sync(0xffffffffu, ic, j0 + h + j) >> 20), 1), be[j]);
            scaled |= (unsigned)(be[j] - 1) >= 2045u;
          }
          if (__any_sync(0xffffffffu, scaled)) {
#pragma unroll
            for (int j = 0; j < 4; ++j)
              if ((unsigned)(be[j] - 1) >= 2045u) v[j] = assemble_scaled(v[j], be[j]);
          }
          if (g.alpha != 1.0) {
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] = g.alpha == -1.0 ? -v[j] : g.alpha * v[j];
          }
          if (g.beta != 0.0) {
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] = g.beta == 1.0 ? v[j] + cv[j] : fma(g.beta, cv[j], v[j]);
          }
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if ((wr >> j) & 1u) cp[g.ldc * j] = v[j];
        }
#pragma unroll
        for (int j = 0; j < EC - 8; ++j) { hi[j] = hi[j + 8]; lo[j] = lo[j + 8]; }
      }
      if (special || __any_sync(0xffffffffu, row_special)) {
        for (int j = 0; j < EC && c0 + j < g.N; ++j) {
          const unsigned icj = __shfl_sync(0xffffffffu, ic, j);
          if (inrow && (row_special || icj >= HI_INF)) {
            double v = ia > HI_INF || icj > HI_INF ? __longlong_as_double(0x7FF8000000000000ll)
                                                   : plain_dot(g, t, row, c0 + j);
            v *= g.alpha;
            if (g.beta != 0.0) v = fma(g.beta, C[g.ldc * (c0 + j)], v);
            C[g.ldc * (c0 + j)] = v;
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(TMEM_COLS)
                 : "memory");
}

// C_b = alpha * sum_s W[b][s] + beta * C_b
__global__ void k_tc_reduce(int m, int n, int S, const double* __restrict__ W, double alpha,
                            double beta, double* __restrict__ C, long long ldc, long long sC) {
  const long long total = (long long)m * n;
  const double* Wb = W + (long long)blockIdx.y * S * total;
  double* Cb = C + (long long)blockIdx.y * sC;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    double acc = Wb[i];
    for (int s = 1; s < S; ++s) acc += Wb[(long long)s * total + i];
    const int r = (int)(i % m);
    const long long c = i / m;
    double* cp = Cb + r + ldc * c;
    double v = alpha * acc;
    if (beta != 0.0) v += beta * (*cp);
    *cp = v;
  }
}

size_t plane_bytes(const Operand& o, int kblks) {
  return (size_t)o.batch * o.row_blocks * kblks * o.rb * 64 * NS;
}

// workspace bound per operand: larger operands are taken in row panels
constexpr size_t TC_PANEL_BYTES = (size_t)1 << 31;

// Few tiles and a long k: k is split at chunk boundaries into at most 16 slices.  The rounds of the
// persistent grid times a slice's chunks (plus half a chunk for the epilogue) decide; returned in
// chunks.
double tc_slices(const qk_ctx* ctx, long long tiles, int nch, int& S) {
  double best = 1e300;
  S = 1;
  for (int s = 1; s <= 16 && s <= nch; ++s) {
    if (s > 1 && tiles * s > 4LL * ctx->num_sms) break;
    const double rounds = (double)((tiles * s + ctx->num_sms - 1) / ctx->num_sms);
    const double cost = rounds * ((nch + s - 1) / s + 0.5) + (s > 1 ? 0.5 : 0.0);
    if (cost < best) { best = cost; S = s; }
  }
  return best;
}

// (QK_ERR_NOMEM before anything has been launched)
int tc_panel(qk_ctx* ctx, TcGemm g) {
  auto finish = [&](Operand& o, int rb) {
    o.rb = rb;
    o.row_blocks = (o.rows + rb - 1) / rb;
    o.batch = o.stride || o.kscale ? g.batch : 1;
  };
  finish(g.a, TM);
  finish(g.b, TN);
  g.kblks = (g.K + KB - 1) / KB;
  g.mt = g.a.row_blocks;
  g.nt = g.b.row_blocks;
  const size_t na = (size_t)g.a.batch * g.a.row_blocks * TM, nb = (size_t)g.b.batch * g.b.row_blocks * TN;
  QK_TRY(qk_wst(ctx, W_TCA, plane_bytes(g.a, g.kblks), &g.a.P));
  QK_TRY(qk_wst(ctx, W_TCB, plane_bytes(g.b, g.kblks), &g.b.P));
  auto slabs = [&](const Operand& o) {
    return g.K <= SELF_K ? 0 : (g.K + (o.trans ? 1023 : 255)) / (o.trans ? 1024 : 256);
  };
  g.a.slabs = slabs(g.a);
  g.b.slabs = slabs(g.b);
  QK_TRY(qk_wst(ctx, W_TCI, na * (1 + g.a.slabs) + nb * (1 + g.b.slabs), &g.a.info));
  g.b.info = g.a.info + na;
  g.a.part = g.b.info + nb;
  g.b.part = g.a.part + na * g.a.slabs;
  const int nch = (g.kblks + CHUNK - 1) / CHUNK;
  const long long tiles = (long long)g.mt * g.nt * g.batch;
  int S = 1;
  if (!g.lower) tc_slices(ctx, tiles, nch, S);
  const int cps = (nch + S - 1) / S;
  S = (nch + cps - 1) / cps;
  g.slices = S;
  g.kb_per_slice = cps * CHUNK;
  const long long units = tiles * S;
  if (units > 0x7fffffffLL) return qk_fail(ctx, QK_ERR_ARG, "tensor-core GEMM: too many tiles");
  const double alpha = g.alpha, beta = g.beta;
  double* C = g.C;
  const long long ldc = g.ldc, sC = g.sC;
  if (S > 1) {
    double* W = nullptr;
    QK_TRY(qk_wst(ctx, W_SPLITK, (size_t)S * g.M * g.N * g.batch, &W));
    g.alpha = 1.0;
    g.beta = 0.0;
    g.C = W;
    g.ldc = g.M;
    g.sC = (long long)g.M * g.N;
  }
  auto strips = [](const Operand& o) { return (o.rows + (o.trans ? 7 : 31)) / (o.trans ? 8 : 32); };
  if (g.K > SELF_K) {
    const int ab = strips(g.a) * g.a.slabs * g.a.batch, bb = strips(g.b) * g.b.slabs * g.b.batch;
    k_tc_rowmax<<<ab + bb, 256, 0, ctx->stream>>>(g.a, g.b, g.K, ab);
    QK_LAUNCHED();
  }
  const int per = g.K <= SELF_K ? 1 : g.kblks;             // blocks of k per strip of 32 rows
  const int sa = g.a.row_blocks * (TM / 32) * per * g.a.batch;
  const int sb = g.b.row_blocks * (TN / 32) * per * g.b.batch;
  if (g.K <= SELF_K) k_tc_slice<true><<<sa + sb, 128, 0, ctx->stream>>>(g.a, g.b, g.K, g.kblks, sa);
  else k_tc_slice<false><<<sa + sb, 128, 0, ctx->stream>>>(g.a, g.b, g.K, g.kblks, sa);
  QK_LAUNCHED();
  static std::once_flag once;
  static cudaError_t attr_err = cudaSuccess;
  std::call_once(once, [] {
    attr_err = cudaFuncSetAttribute(k_gemm_tc, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    SMEM_BYTES);
  });
  QK_CK(attr_err);
  const int grid = (int)(units < ctx->num_sms ? units : ctx->num_sms);
  k_gemm_tc<<<grid, NTHREADS, SMEM_BYTES, ctx->stream>>>(g, ctx->d_status);
  QK_LAUNCHED();
  if (S > 1) {
    long long blocks = ((long long)g.M * g.N + 255) / 256;
    if (blocks > 8 * ctx->num_sms) blocks = 8 * ctx->num_sms;
    k_tc_reduce<<<dim3((unsigned)blocks, g.batch), 256, 0, ctx->stream>>>(g.M, g.N, S, g.C, alpha,
                                                                       beta, C, ldc, sC);
    QK_LAUNCHED();
  }
  return QK_OK;
}

}  // namespace

int qk_gemm_tc(qk_ctx* ctx, char ta, char tb, int m, int n, int k, double alpha, const double* A,
               long long lda, long long strideA, const double* B, long long ldb, long long strideB,
               double beta, double* C, long long ldc, long long strideC, int batch, bool always) {
  return qk_gemm_tc_ex(ctx, ta, tb, m, n, k, alpha, A, lda, strideA, B, ldb, strideB, nullptr, 0, beta, C,
                       ldc, strideC, batch, false, always);
}

int qk_gemm_tc_basis(qk_ctx* ctx, char ta, char tb, int m, int n, int k, double alpha, const double* A,
                     long long lda, const double* B, long long ldb, double beta, double* C,
                     long long ldc, qk_basis_exp* be) {
  return qk_gemm_tc_ex(ctx, ta, tb, m, n, k, alpha, A, lda, 0, B, ldb, 0, nullptr, 0, beta, C, ldc, 0, 1,
                       false, false, be);
}

int qk_gemm_tc_ex(qk_ctx* ctx, char ta, char tb, int m, int n, int k, double alpha, const double* A,
                  long long lda, long long strideA, const double* B, long long ldb, long long strideB,
                  const double* kscale, long long sK, double beta, double* C, long long ldc,
                  long long strideC, int batch, bool lower, bool always, qk_basis_exp* be) {
  if (m <= 0 || n <= 0 || batch <= 0) return QK_OK;
  if (kscale && !always) return qk_fail(ctx, QK_ERR_ARG, "scaled GEMM: tensor-core path only");
  if (!always && lower && !qk_gemm_tc_pays(ctx, m, n / 2 + 1, k, batch))
    return qk_dgemm_lower(ctx, ta, tb, m, n, k, alpha, A, lda, strideA, B, ldb, strideB, beta, C, ldc,
                          strideC, batch);
  // (k below 2^20 keeps the integer sums within 95 bits)
  if (kscale && (k <= 0 || k > (1 << 20))) return qk_fail(ctx, QK_ERR_ARG, "scaled GEMM: k=%d", k);
  if (k <= 0 || k > (1 << 20) || !(always || lower || qk_gemm_tc_pays(ctx, m, n, k, batch)))
    return qk_dgemm(ctx, ta, tb, m, n, k, alpha, A, lda, strideA, B, ldb, strideB, beta, C, ldc,
                    strideC, batch);
  const bool TA = (ta == 'T' || ta == 't'), TB = (tb == 'T' || tb == 't');
  TcGemm g = {};
  g.K = k;
  g.alpha = alpha;
  g.beta = beta;
  g.ldc = ldc;
  g.sC = strideC;
  if (be) {
    if (!be->e) {
      int* kexp = nullptr;
      const int st = qk_wst(ctx, W_TCK, (size_t)k, &kexp);
      if (qk_oom_dropped(ctx, st))
        return qk_dgemm(ctx, ta, tb, m, n, k, alpha, A, lda, strideA, B, ldb, strideB, beta, C, ldc,
                        strideC, batch);
      QK_TRY(st);
      g.b.X = be->c;
      g.b.ld = be->ld;
      g.b.rows = be->n;
      g.b.trans = 1;
      k_tc_kexp<<<(k + 7) / 8, 256, 0, ctx->stream>>>(g.b, k, kexp);
      QK_LAUNCHED();
      be->e = kexp;
    }
    g.a.kexp = g.b.kexp = be->e;
    g.b.kneg = 1;
  }
  const size_t row_bytes = (size_t)((k + KB - 1) / KB) * 64 * NS;
  // batch entries per launch: the planes of one operand within the bound (and grid.y of the split-K
  // reduction); then row panels where a single entry exceeds it.  The lower form takes square panels:
  // those on the diagonal in that form, those below it whole
  const size_t bound = ctx->tc_panel_kb > 0 ? (size_t)ctx->tc_panel_kb << 10 : TC_PANEL_BYTES;
  const size_t entry = row_bytes * (size_t)(m > n ? m : n);
  long long b_step = (long long)(bound / entry);
  b_step = b_step < 1 ? 1 : (b_step > 65535 ? 65535 : b_step);
  if (b_step > batch) b_step = batch;
  auto panel = [&](int rows, int rb) {
    long long p = (long long)(bound / row_bytes) / rb * rb;
    if (p < rb) p = rb;
    return p < rows ? (int)p : rows;
  };
  int pm = b_step > 1 ? m : panel(m, TM), pn = b_step > 1 ? n : panel(n, TN);
  if (lower && (pm < m || pn < n)) pm = pn = panel(m > n ? m : n, TM);
  for (int b0 = 0; b0 < batch; b0 += (int)b_step)
    for (int j0 = 0; j0 < n; j0 += pn)
      for (int i0 = lower ? j0 : 0; i0 < m; i0 += pm) {
        g.lower = lower && i0 == j0 ? 1 : 0;
        g.batch = batch - b0 < b_step ? batch - b0 : (int)b_step;
        g.M = m - i0 < pm ? m - i0 : pm;
        g.N = n - j0 < pn ? n - j0 : pn;
        g.a.X = A + b0 * strideA + (TA ? (long long)i0 * lda : i0);
        g.a.ld = lda;
        g.a.stride = batch > 1 ? strideA : 0;
        g.a.rows = g.M;
        g.a.trans = TA;
        g.b.X = B + b0 * strideB + (TB ? j0 : (long long)j0 * ldb);
        g.b.kscale = kscale ? kscale + b0 * sK : nullptr;
        g.b.sk = sK;
        g.b.ld = ldb;
        g.b.stride = batch > 1 ? strideB : 0;
        g.b.rows = g.N;
        g.b.trans = !TB;
        g.C = C + b0 * strideC + i0 + (long long)j0 * ldc;
        const int st = tc_panel(ctx, g);
        // no room for the digit planes: the FMA kernel needs none
        if (!kscale && qk_oom_dropped(ctx, st))
          QK_TRY((g.lower ? qk_dgemm_lower : qk_dgemm)(ctx, ta, tb, g.M, g.N, k, alpha, g.a.X, lda, strideA,
                                                       g.b.X, ldb, strideB, beta, g.C, ldc, strideC,
                                                       g.batch));
        else QK_TRY(st);
      }
  return QK_OK;
}

// Whether the tensor-core path is the faster one for this product.  Both costs are in
// microseconds on one GB300: DFMA runs its 16 x 16 tiles at ~1.1 TFLOP/s; a 128 x 64 x 128 chunk on
// the tensor cores takes ~7.2 us per SM and a tile's k is spread over 16 SMs at most, the operands'
// preparation moves 32 bytes an element, and its launches and their latency cost ~15 us against ~5
// (measured, DFMA / tensor cores: 128 x 128 x 400 16 / 30 us, 400 x 128 x 128 14 / 22, 567 x 128 x 128
// 20 / 23, 128 x 400 x 400 45 / 33, 400 x 400 x 128 46 / 24; with a call's 22 us: 48 x 48 x 15360 92 /
// 113, 64 x 64 x 4096 58 / 60, 64 x 64 x 32768 288 / 195, 20 x 20 x 200000 460 / 951).
bool qk_gemm_tc_pays(const qk_ctx* ctx, int m, int n, int k, int batch) {
  if (k < 16) return false;
  const double pm = (m + 15) / 16 * 16.0, pn = (n + 15) / 16 * 16.0;
  const double dfma = 5.0 + 2.0 * pm * pn * k * batch / 1.1e6;
  const long long tiles = (long long)((m + TM - 1) / TM) * ((n + TN - 1) / TN) * batch;
  int S;
  const double chunks = tc_slices(ctx, tiles, (k + 127) / 128, S);
  const double tc = 15.0 + 7.2 * (chunks - 0.5) + ((double)m + n) * k * batch * 32.0 / 4e6;
  return tc < dfma;
}

// Montgomery arithmetic on 52-bit digits held as doubles, for integers spread
// over TPI lanes with D digits per lane (lane g: digits gD .. gD + D - 1;
// N = TPI * D digits, R = 2^(52 N)).
//
// The product of two digits comes from the FP64 pipe exactly, as two halves
// on a 2^52 grid (the fused multiply-add splitting of N. Emmart, F. Zheng and
// C. Weems, "Faster modular exponentiation using double precision floating
// point arithmetic on the GPU", ARITH 2018):
//   h = fma_rz(a, b, 1.5 * 2^104)           floor(ab / 2^52) in h's low mantissa bits
//   l = fma_rz(a, b, (1.5 * 2^104 + 2^52) - h)   ab mod 2^52 in l's
// and both are added to 64-bit columns as the doubles' own bits, so a digit
// product costs three FP64 operations and two 64-bit adds and nothing carries
// between columns inside a product: the exponent bits of every h and l are
// constants whose sum per column is known and is subtracted once at the end.
// Why it is faster than rows of 32-bit limbs (mont.cuh): measured on B200, one
// 52 x 52-bit product takes 9.9 cycles of a scheduler where one 32 x 32-bit
// product of a mul.wide row with its two carry chains takes 5.9: 273 against
// 174 bit-by-bit products a lane and cycle.  Both are bound by operand delivery (the FP64
// instructions read 64-bit registers; ncu: issue slots half empty, stalls
// "math pipe throttle" and "dispatch"), not by the FP64 rate.
//
// Digits are balanced, |d| <= 2^51 + 2^12, so that 1.5 * 2^104 + ab stays in
// one binade; values are signed and almost reduced, |v| <= N (the modulus):
// |ab| / R + N / 2 <= N since R >= 4 N, so no product needs a subtraction and
// the carries left at its end are pushed one digit up and no further.
#pragma once
#include "internal.h"
#include "mont.cuh"

namespace xmpb {

constexpr double kDigHi = 0x1.8p104;              // splits off multiples of 2^52
constexpr double kDigLo = 0x1.8p104 + 0x1p52;     // minus h: leaves the low half on 2^52
constexpr uint64_t kDigMask = (1ull << 52) - 1;
// Exponent bits a column collects, in units of its bits 52 and up: 0x433 per low half; per high half
// 0x467 and half a unit (the 0.5 of 1.5 * 2^104 is mantissa bit 51).  High halves come in pairs.
constexpr uint32_t kDigLoBits = 0x433u, kDigHiPairBits = 2u * 0x467u + 1u;

// Digits per lane of TPI lanes that hold 32 * TPI * L bits with two bits to spare (R >= 4 N).
__host__ __device__ constexpr int dig_count(int TPI, int L) { return (32 * TPI * L + 2 + 52 * TPI - 1) / (52 * TPI); }

__device__ __forceinline__ uint64_t dig_bits(double v) { return (uint64_t)__double_as_longlong(v); }

// col[O + j] += low half, col[O + j + 1] += high half of a[j] * w.  All first
// steps, then all second, then all third: the steps of one product depend on
// each other (about eight cycles each), so a lane needs the other products in
// between.
template <int D, int O, int C>
__device__ __forceinline__ void dig_row(uint64_t (&col)[C], const double (&a)[D], double w) {
  double h[D], t[D];
#pragma unroll
  for (int j = 0; j < D; j++) h[j] = __fma_rz(a[j], w, kDigHi);
#pragma unroll
  for (int j = 0; j < D; j++) t[j] = __dsub_rn(kDigLo, h[j]);
#pragma unroll
  for (int j = 0; j < D; j++) t[j] = __fma_rz(a[j], w, t[j]);
#pragma unroll
  for (int j = 0; j < D; j++) {
    col[O + j] += dig_bits(t[j]);
    col[O + j + 1] += dig_bits(h[j]);
  }
}

template <int TPI>
__device__ __forceinline__ double dig_bcast(double v, int src) {
  if (TPI == 1) return v;
  return __hiloint2double(__shfl_sync(kFull, __double2hiint(v), src, TPI),
                          __shfl_sync(kFull, __double2loint(v), src, TPI));
}

// This warp's operand B in shared memory: digit p of group i at p * (32 / TPI) + i, so that the groups
// of a warp read a digit as neighbouring words.  32 * D doubles a warp; also the staging area between
// limbs and digits.
struct DigSmem {
  double *b;
};
template <int TPI, int D>
__device__ __forceinline__ double *dig_b(const DigSmem &s) {
  return s.b + (threadIdx.x & 31) / TPI;
}
// Stores this lane's digits as operand B (all lanes of the warp call it together).
template <int TPI, int D>
__device__ __forceinline__ void dig_set_b(const Group<TPI> &G, const DigSmem &s, const double (&x)[D]) {
  __syncwarp();
  double *b = dig_b<TPI, D>(s) + (size_t)G.lane * D * (32 / TPI);
#pragma unroll
  for (int j = 0; j < D; j++) b[j * (32 / TPI)] = x[j];
  __syncwarp();
}

// Columns (true sum of column j = col[j] - kbits[j] * 2^52, signed) to balanced digits: each keeps its
// low 52 bits as a balanced digit and passes the rest to the next one, once.  `khi` is the constant of
// this lane's column 0 in the high word, falling by `kstep` per column.  The value's top digit passes
// nothing on (its value is within +-R / 4).
template <int TPI, int D, int C>
__device__ __forceinline__ void dig_settle(const Group<TPI> &G, double (&r)[D], const uint64_t (&col)[C], uint32_t khi,
                                           uint32_t kstep) {
  uint32_t up[D];  // carry + 2048
#pragma unroll
  for (int j = 0; j < D; j++) {
    // + 2^51 (balanced) and + 2048 * 2^52 (carry as an unsigned field)
    const uint32_t u = (uint32_t)(col[j] >> 32) - (khi - (uint32_t)j * kstep) + 0x80080000u;
    up[j] = u >> 20;
    r[j] = __dsub_rn(__hiloint2double((int)((u & 0xfffffu) | 0x43300000u), (int)(uint32_t)col[j]),
                     0x1p53 + 0x1p51 + 2048.0);
  }
  uint32_t in = 2048u;
  if (TPI > 1) {
    in = __shfl_up_sync(kFull, up[D - 1], 1, TPI);
    if (G.lane == 0) in = 2048u;
  }
#pragma unroll
  for (int j = 0; j < D; j++) r[j] = __dadd_rn(r[j], __hiloint2double(0x43300000, (int)(j ? up[j ? j - 1 : 0] : in)));
}

// Rows a step of dig_mul unrolls; the exponentiation loop's code must fit the instruction cache: all of
// them up to ten digits without the square (4 x 16, ten rows: 21.6 ms; five 21.6 and a lone instance 3.2
// instead of 3.0 ms), five with it (1 x 16 4.92 / 4.88 ms; 1 x 32 22.7 / 21.5) and at fifteen digits (4 x 24
// 54.0 / 46.7 ms), two at twenty (2 x 32: 57.1 ms with all, 42.1 with five, 40.5).
__host__ __device__ constexpr int dig_mul_step(int TPI, int D) {
  return D == 20 && TPI > 1 ? 2 : D == 15 || D == 20 || (TPI == 1 && D == 10) ? 5 : D;
}

// r = a * B * R^-1 mod N (|r| <= N), B the operand in shared memory.  n: the
// modulus's digits; np = -N^-1 mod 2^52 (lane 0's is used).  r may alias a.
// A row adds a * b_i and n * q with q fixing column 0 mod 2^52, and drops that
// column: its carry goes to lane 0's next column, and every other lane's
// column 0 moves to the top of the lane below.  The columns do not carry, so
// the order of the additions is free: a * b_(i+1) is added between the
// quotient digit and the products that wait for it, which hides the digit's
// latency (a lone 1024-bit chain on 4 lanes: 3.25 -> 2.15 us a product).
// The shift is register renaming inside a step of U rows and D + 2 register moves from step to step.
template <int TPI, int D>
__device__ __forceinline__ void dig_mul(const Group<TPI> &G, double (&r)[D], const double (&a)[D], const DigSmem &sm,
                                        const double (&n)[D], uint64_t np) {
  constexpr int N = TPI * D, STEP = 32 / TPI, U = dig_mul_step(TPI, D);
  const double *bp = dig_b<TPI, D>(sm);
  uint64_t col[D + 2];
#pragma unroll
  for (int j = 0; j < D + 2; j++) col[j] = 0;
  uint32_t k = 2u * kDigLoBits << 20;  // the constant of the column that row i drops, in its high word
  const uint32_t lane0 = G.lane == 0 ? kFull : 0u;
  dig_row<D, 0>(col, a, bp[0]);
#pragma unroll 1
  for (int i = 0; i < N; i += U) {
#pragma unroll
    for (int row = 0; row < U; row++) {
      const uint64_t x = col[0] * np;
      double q = __dsub_rn(__hiloint2double((int)(((uint32_t)(x >> 32) & 0xfffffu) ^ 0x43380000u), (int)(uint32_t)x),
                           0x1.8p52);  // low 52 bits, balanced
      q = dig_bcast<TPI>(q, 0);
      if (row + 1 < U || i + U < N) dig_row<D, 1>(col, a, bp[(i + row + 1) * STEP]);
      dig_row<D, 0>(col, n, q);
      int32_t c = (int32_t)((uint32_t)(col[0] >> 32) - k) >> 20;
      k += (2u * kDigLoBits + kDigHiPairBits) << 20;
      uint64_t next = 0;
      if (TPI > 1) {
        c &= (int32_t)lane0;
        const uint32_t lo = __shfl_down_sync(kFull, (uint32_t)col[0], 1, TPI);
        const uint32_t hi = __shfl_down_sync(kFull, (uint32_t)(col[0] >> 32), 1, TPI);
        next = G.lane == TPI - 1 ? 0ull : ((uint64_t)hi << 32) | lo;
      }
#pragma unroll
      for (int j = 0; j <= D; j++) col[j] = col[j + 1];
      col[D + 1] = 0;
      col[D - 1] += next;
      col[0] += (uint64_t)(int64_t)c;
    }
  }
  // column p collected 2 (N - 1 - p) low and N - p pairs of high halves
  const uint32_t p0 = G.lane * D;
  dig_settle<TPI, D>(G, r, col, (2u * (N - 1 - p0) * kDigLoBits + (N - p0) * kDigHiPairBits) << 20,
                     (2u * kDigLoBits + kDigHiPairBits) << 20);
}

// ---- squares, one lane an instance ----------------------------------------------------
//
// r = a^2 R^-1: the square's 2D columns first, each digit product a_i a_j (i < j) once and doubled, then the
// reduction's rows n * q alone on them: D (D + 1) / 2 + D^2 digit products instead of 2 D^2.  Columns start
// from minus the constant of the halves they will take, so the reduction's constants are its own.
constexpr uint64_t kDigLoBits64 = (uint64_t)kDigLoBits << 52, kDigHiBits64 = (0x467ull << 52) + (1ull << 51);
// Digit pairs (i, j), i < j < D, with i + j = c.
__host__ __device__ constexpr int dig_cross_pairs(int c, int D) {
  const int lo = c - D + 1 > 0 ? c - D + 1 : 0, end = (c + 1) / 2;
  return c < 0 || end < lo ? 0 : end - lo;
}
// Half the constant of column c of a square of D digits formed as twice its cross products plus its squares.
__host__ __device__ constexpr uint64_t dig_square_const(int c, int D) {
  return (uint64_t)dig_cross_pairs(c, D) * kDigLoBits64 + (uint64_t)dig_cross_pairs(c - 1, D) * kDigHiBits64 +
         (c % 2 ? kDigHiBits64 : kDigLoBits64) / 2;
}

// s = the 2D columns of a^2, as true signed sums.
template <int D>
__device__ __forceinline__ void dig_block_square(uint64_t (&s)[2 * D], const double (&a)[D]) {
#pragma unroll
  for (int c = 0; c < 2 * D; c++) s[c] = 0 - dig_square_const(c, D);
#pragma unroll
  for (int i = 0; i + 1 < D; i++) {
    double h[D], t[D];
#pragma unroll
    for (int j = i + 1; j < D; j++) h[j] = __fma_rz(a[i], a[j], kDigHi);
#pragma unroll
    for (int j = i + 1; j < D; j++) t[j] = __dsub_rn(kDigLo, h[j]);
#pragma unroll
    for (int j = i + 1; j < D; j++) t[j] = __fma_rz(a[i], a[j], t[j]);
#pragma unroll
    for (int j = i + 1; j < D; j++) {
      s[i + j] += dig_bits(t[j]);
      s[i + j + 1] += dig_bits(h[j]);
    }
  }
  double h[D], t[D];
#pragma unroll
  for (int j = 0; j < D; j++) h[j] = __fma_rz(a[j], a[j], kDigHi);
#pragma unroll
  for (int j = 0; j < D; j++) t[j] = __dsub_rn(kDigLo, h[j]);
#pragma unroll
  for (int j = 0; j < D; j++) t[j] = __fma_rz(a[j], a[j], t[j]);
#pragma unroll
  for (int j = 0; j < D; j++) {
    s[2 * j] = 2 * s[2 * j] + dig_bits(t[j]);
    s[2 * j + 1] = 2 * s[2 * j + 1] + dig_bits(h[j]);
  }
}

// r = a^2 R^-1 mod N (|r| <= N).  r may alias a.  A row makes column 0 of what is left 0 mod 2^52 and drops it;
// k is the high word of the constant that the halves of n * q have left in it (the low word stays 0).
template <int D>
__device__ __forceinline__ void dig_sqr1(const Group<1> &G, double (&r)[D], const double (&a)[D], const double (&n)[D],
                                         uint64_t np) {
  uint64_t col[2 * D];
  dig_block_square<D>(col, a);
  uint32_t k = 0;
  constexpr uint32_t kstep = (uint32_t)((kDigLoBits64 + kDigHiBits64) >> 32);
#pragma unroll
  for (int row = 0; row < D; row++) {
    const uint64_t x = (((uint64_t)((uint32_t)(col[0] >> 32) - k) << 32) | (uint32_t)col[0]) * np;
    const double q = __dsub_rn(
        __hiloint2double((int)(((uint32_t)(x >> 32) & 0xfffffu) ^ 0x43380000u), (int)(uint32_t)x), 0x1.8p52);
    dig_row<D, 0>(col, n, q);
    const int32_t c = (int32_t)((uint32_t)(col[0] >> 32) - k - (kDigLoBits << 20)) >> 20;
    k += kstep;
#pragma unroll
    for (int j = 0; j < 2 * D - 1; j++) col[j] = col[j + 1];
    col[0] += (uint64_t)(int64_t)c;
  }
  // column p collected D - 1 - p low and D - p high halves of n * q
  dig_settle<1, D>(G, r, col, (uint32_t)(((D - 1) * kDigLoBits64 + D * kDigHiBits64) >> 32), kstep);
}

// ---- limbs <-> digits ----------------------------------------------------------------

// Balanced digits of this lane from limb(j) (zero above the number): digit p is the 52 bits at 52 p,
// less 2^52 if its top bit is set, plus the top bit of the digit below.  `first`: the number's digit
// that is the group's digit 0 (a number of two N digits is taken in two parts).
template <int TPI, int D, class Limb>
__device__ __forceinline__ void dig_from_limbs(const Group<TPI> &G, double (&x)[D], Limb limb, uint32_t first = 0) {
  uint32_t below = 0;
  {
    const uint32_t o = 52 * (first + G.lane * D);
    if (o) below = (limb((o - 1) >> 5) >> ((o - 1) & 31)) & 1u;
  }
#pragma unroll
  for (int j = 0; j < D; j++) {
    const uint32_t o = 52 * (first + G.lane * D + j), w = o >> 5, s = o & 31;
    const uint64_t lo = (uint64_t)limb(w + 1) << 32 | limb(w);
    uint64_t v = lo >> s;
    if (s) v |= (uint64_t)limb(w + 2) << (64 - s);
    v &= kDigMask;
    const uint32_t top = (uint32_t)(v >> 51);
    x[j] = (double)((int64_t)v - ((int64_t)top << 52) + (int64_t)below);
    below = top;
  }
}

// Digits of element e of an integer array.
template <int TPI, int D>
__device__ __forceinline__ void dig_load(const Group<TPI> &G, double (&x)[D], const uint32_t *limbs, uint32_t nlimbs,
                                         uint32_t stride, uint32_t e, uint32_t first = 0) {
  dig_from_limbs<TPI, D>(G, x, [&](uint32_t j) { return load_limb(limbs, nlimbs, stride, e, j); }, first);
}

// Digits from limbs held as TPI lanes x L limbs, through this warp's shared memory.
template <int TPI, int L, int D>
__device__ __forceinline__ void dig_from_lanes(const Group<TPI> &G, double (&x)[D], const uint32_t (&v)[L],
                                               const DigSmem &sm) {
  uint32_t *st = reinterpret_cast<uint32_t *>(sm.b) + (size_t)((threadIdx.x & 31) / TPI) * (TPI * L);
  __syncwarp();
#pragma unroll
  for (int k = 0; k < L; k++) st[G.lane * L + k] = v[k];
  __syncwarp();
  dig_from_limbs<TPI, D>(G, x, [&](uint32_t j) { return j < (uint32_t)(TPI * L) ? st[j] : 0u; });
  __syncwarp();
}

// Carries the signed digits d into [0, 2^52) across the group (the same steps
// whatever their values); returns the carry out of the top lane (-1: the value
// was negative, 0 otherwise for |value| < R).
template <int TPI, int D>
__device__ __forceinline__ int32_t dig_carry(const Group<TPI> &G, int64_t (&d)[D]) {
  int32_t in = 0, total = 0;
#pragma unroll 1
  for (int pass = 0; pass < TPI; pass++) {
    int64_t c = in;
#pragma unroll
    for (int j = 0; j < D; j++) {
      const int64_t t = d[j] + c;
      d[j] = t & (int64_t)kDigMask;
      c = t >> 52;
    }
    total += (int32_t)c;
    if (TPI > 1) {
      in = __shfl_up_sync(kFull, (int32_t)c, 1, TPI);
      if (G.lane == 0) in = 0;
    }
  }
  return TPI == 1 ? total : __shfl_sync(kFull, total, TPI - 1, TPI);
}

// c = the digits of v mod N in [0, N) for |v| < N, as 52-bit integers.
template <int TPI, int D>
__device__ __forceinline__ void dig_canon(const Group<TPI> &G, int64_t (&c)[D], const double (&v)[D],
                                          const double (&n)[D]) {
#pragma unroll
  for (int j = 0; j < D; j++) c[j] = (int64_t)v[j];
  const bool neg = dig_carry<TPI, D>(G, c) < 0;
#pragma unroll
  for (int j = 0; j < D; j++) c[j] += neg ? (int64_t)n[j] : 0;
  dig_carry<TPI, D>(G, c);
}

// Group g (four limbs) of the number whose 52-bit digits are d[0 .. count), zero above.
__device__ __forceinline__ uint4 dig_group(const uint64_t *d, uint32_t count, uint32_t g) {
  uint64_t w[2];
#pragma unroll
  for (int half = 0; half < 2; half++) {
    const uint32_t o = 128 * g + 64 * half, p = o / 52, s = o % 52;
    const uint64_t d0 = p < count ? d[p] : 0, d1 = p + 1 < count ? d[p + 1] : 0, d2 = p + 2 < count ? d[p + 2] : 0;
    w[half] = d0 >> s | d1 << (52 - s);
    if (s > 40) w[half] |= d2 << (104 - s);
  }
  return make_uint4((uint32_t)w[0], (uint32_t)(w[0] >> 32), (uint32_t)w[1], (uint32_t)(w[1] >> 32));
}

// Stores canonical digits to element o of `out` (limbs above the digits as zero).
template <int TPI, int D>
__device__ __forceinline__ void dig_store(const Group<TPI> &G, const int64_t (&c)[D], const OutView &out, uint32_t o,
                                          bool valid, const DigSmem &sm) {
  uint64_t *st = reinterpret_cast<uint64_t *>(sm.b) + (size_t)((threadIdx.x & 31) / TPI) * (TPI * D);
  __syncwarp();
#pragma unroll
  for (int j = 0; j < D; j++) st[G.lane * D + j] = (uint64_t)c[j];
  __syncwarp();
  if (valid && o < out.count)
    for (uint32_t g = G.lane; g < div_up(out.nlimbs, 4); g += TPI)
      store_group(out.limbs, out.nlimbs, out.stride, o, g, dig_group(st, TPI * D, g));
  __syncwarp();
}

// ---- constants of a modulus -----------------------------------------------------------

// -N^-1 mod 2^64 from the two lowest limbs (lane 0's is the group's), N odd: Newton's iteration from
// three correct bits.
__device__ __forceinline__ uint64_t dig_neg_inv(uint32_t n0, uint32_t n1) {
  const uint64_t n = (uint64_t)n1 << 32 | n0;
  uint64_t x = n;
#pragma unroll
  for (int i = 0; i < 5; i++) x = x * (2 - n * x);
  return 0 - x;
}

// r2 = R^2 mod N (|r2| <= N), N odd, given as limbs nl (TPI lanes x L) and digits n.  2^(bitlen N - 1) is
// doubled exactly on the limbs up to 2^(52N + s), 52N = s 2^j with s odd: Montgomery form of 2^s, which j
// squarings bring to that of 2^(52N) = R.  (With limbs R = 2^(32n): one doubling and 11 squarings at 2048
// bits; here 98 doublings, about two products' time, and 5.)  N = 1 gives 0.
template <int TPI, int L, int D>
__device__ __forceinline__ void dig_r2(const Group<TPI> &G, double (&r2)[D], const uint32_t (&nl)[L],
                                       const double (&n)[D], uint64_t np, const DigSmem &sm) {
  constexpr uint32_t bits = 52u * TPI * D;
  const uint32_t j = __ffs(bits) - 1, s = bits >> j;
  const uint32_t b = dbitlen<TPI, L>(G, nl);
  const bool trivial = b <= 1;
  const uint32_t tb = trivial ? 0u : b - 1;
  uint32_t v[L];
#pragma unroll
  for (int k = 0; k < L; k++) v[k] = !trivial && (G.lane * L + k) == (tb >> 5) ? 1u << (tb & 31) : 0u;
  const uint32_t doublings = trivial ? 0u : bits + s - tb;
  const uint32_t dmax = __reduce_max_sync(kFull, doublings);
#pragma unroll 1
  for (uint32_t i = 0; i < dmax; i++) dmod_double<TPI, L>(G, v, nl, i < doublings);
  dig_from_lanes<TPI, L, D>(G, r2, v, sm);
#pragma unroll 1
  for (uint32_t q = 0; q < j; q++) {
    dig_set_b<TPI, D>(G, sm, r2);
    dig_mul<TPI, D>(G, r2, r2, sm, n, np);
  }
}

// Digits per lane when the kernel of this shape multiplies on 52-bit digits, 0 when on 32-bit limbs
// (mont.cuh).  Every registered shape was timed both ways on B200 (512-bit exponents; 151,552 / TPI
// instances, a quarter and a sixteenth of that, and one; limbs / digits): from six limbs a lane on the
// digits are faster throughout (2048 bits, 4 x 16: 36.6 / 21.8 ms, one instance 4.73 / 3.03 ms; 4 x 8:
// 10.3 / 6.7 ms; 8 x 12: 42.9 / 29.4 ms; 1 x 8: 1.13 / 0.85 ms; 16 x 6, 22.5 / 17.9 ms, is the least),
// below that the few digits hold too much padding (4 x 4: three digits a lane for 128 bits, 1.0x at the
// full batch and 0.76x at a sixteenth; 16 x 3: 1.18x and 0.88x; 8 x 5: 0.9x; 1 x 5: 0.95x).
__host__ __device__ constexpr int powm_digits(int TPI, int L) {
  return L >= 6 ? dig_count(TPI, L) : 0;
}

// Words per lane of one window-table entry.
__host__ __device__ constexpr int powm_slot_words(int TPI, int L) {
  return powm_digits(TPI, L) ? 2 * powm_digits(TPI, L) : L;
}

// log2 of the kernel's Montgomery radix (what a precomputed R^2 mod N belongs to).
__host__ __device__ constexpr uint32_t powm_radix_bits(int TPI, int L) {
  return powm_digits(TPI, L) ? 52u * TPI * powm_digits(TPI, L) : 32u * TPI * L;
}

// Whether the digit kernel squares with dig_sqr1.  Measured against the same kernels squaring with dig_mul:
// 256 bits 0.85 -> 0.77 ms (151,552 instances, 512-bit exponents), 512 bits 5.6 -> 4.9, 768 bits 13.3 ->
// 11.4, 1024 bits 28 -> 21.5; one 512-bit instance 0.77 -> 0.66 ms.  Over two and four
// lanes the same saving (each lane its block's square, the block pairs shared out, columns through the
// thread's shared memory) measured no faster at a full batch and slower below (2 x 16: 1.73x against 1.71x of
// the limb kernel's rate at the full batch, 1.29x against 1.58x for one instance; 4 x 16: 1.64x / 1.68x and
// 1.27x / 1.56x): without a * b's products in the rows nothing hides the quotient digits' latency.
__host__ __device__ constexpr bool powm_dig_sqr(int TPI, int L) { return powm_digits(TPI, L) > 0 && TPI == 1; }

}  // namespace xmpb

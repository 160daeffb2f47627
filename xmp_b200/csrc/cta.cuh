// Latency distribution: one exponentiation per CTA.
//
// The lane kernels (powm_kernel.cuh) multiply row by row, each row waiting on
// the previous one's quotient digit: a lone 2048-bit exponentiation takes 7.7 ms
// on them, the floor under a server's latency.  Here a CTA forms a Montgomery
// product as three whole-operand products with no digit-serial dependency
// (Montgomery's REDC on the whole low half):
//   T = a b,   m = (T mod R) N' mod R   (N' = -N^-1 mod R),   U = T + m N,   r = U / R,
// on balanced 52-bit digits in doubles with columns that do not carry
// (dmont.cuh).  P lanes share the columns c and N + c of a product, which
// together have a term for every digit of x: lane p multiplies x_i by
// y_((c - i) mod N), i = p mod P (y is stored twice, so that no index wraps), and
// adds the halves to its sums of one column or the other.  Shuffles add the
// lanes' sums, each step halving the sums that a lane holds; a column is its low
// halves and the high halves of the column below, and one step of carries, each
// column's to the next, makes digits of them.  No resolution is needed because
// operands need not be canonical:
//   - m is only needed mod R, so the carry out of its top digit is dropped;
//   - T's upper columns stay in the lanes' sums, to which m N's are added;
//   - U's low half is a multiple c R of R, so c is read off its two top
//     columns, whatever is below them being far less than half of R.
// Values stay within |v| <= N: |ab| / R + N / 2 since R >= 4 N.  A product is
// three times [terms, barrier, digits, barrier], 300 instructions a warp at 40
// digits, and takes 2,100 cycles: the scheduler issues in 35% of them, the rest
// waits on the chain of FP64 steps, shuffles and barriers.  P sets the length of
// that chain: 2048 bits take 3.53 / 2.56 / 2.95 ms with 4 / 8 / 16 lanes, 4096
// bits 12.8 / 9.75 ms with 4 / 8, 1024 bits 0.99 / 1.01 ms with 4 / 8.  Against
// 4 x 4-word tiles of 32-bit words summed through shared memory and resolved by
// a single warp's ballot lookahead (9 barriers): one exponentiation alone,
// full-length exponents, 1024 bits 1.14 -> 0.99 ms, 2048 bits 3.06 -> 2.56, 3072
// bits 7.82 -> 5.94, 4096 bits 16.9 -> 9.75.  (52-bit digits in tiles through
// shared memory: 0.87, 3.94, 7.57 and 13.1 ms.)  It does not reach the lane
// kernels' throughput, so it serves small batches.
//
// Supported sizes: moduli up to 1024, 2048, 3072, 4096 bits in 20, 40, 60, 80
// digits (any R >= 4 N works).
#pragma once
#include "powm_kernel.cuh"

namespace xmpb {

// LIMBS: the modulus class in limbs (32, 64, 96, 128).
template <int LIMBS>
struct CtaShape {
  static_assert(LIMBS % 32 == 0 && LIMBS >= 32 && LIMBS <= 128, "CTA distribution: 32, 64, 96 or 128 limbs");
  static constexpr int N = LIMBS * 5 / 8;      // digits: 52 N = 32 LIMBS + LIMBS / 2 bits
  static constexpr int P = LIMBS == 32 ? 4 : 8;  // lanes per column pair
  static constexpr int K = (N + P - 1) / P;    // products per lane
  static constexpr int CHUNK = K <= 5 ? K : (K + 1) / 2;  // a warp skips the chunks without terms it needs
  static constexpr int THREADS = (N * P + 31) / 32 * 32;
  static constexpr int PAD = 8;  // words around an operand that the lanes beyond it read and do not use
};

// Shared memory of one CTA (the window table follows it, `entries` x N digits).  Operands of role y are stored
// twice, so that digit (c - i) mod N is at c - i + N.
template <int LIMBS>
struct CtaSmem {
  static constexpr int N = CtaShape<LIMBS>::N, PAD = CtaShape<LIMBS>::PAD;
  uint64_t low[2 * N + 2], high[2 * N + 2];  // column sums of the products' low and high halves, from 2 on
  double pad0[PAD];
  double n[2 * N + PAD], np[2 * N + PAD];  // modulus, -N^-1 mod R
  double acc[2 * N + PAD], x[2 * N + PAD];
  double t[N + PAD], m[N + PAD], one[N + PAD];  // T mod R; m
};

template <int LIMBS>
__host__ __device__ constexpr uint32_t cta_smem_bytes(uint32_t entries) {
  static_assert(sizeof(CtaSmem<LIMBS>) % 16 == 0, "the window table follows");
  return (uint32_t)sizeof(CtaSmem<LIMBS>) + (entries * CtaShape<LIMBS>::N + CtaShape<LIMBS>::PAD) * 8;
}

// This thread's place: lane p of the group of columns c and N + c; and, as a thread of the first N, digit d.
template <int LIMBS>
struct CtaPlace {
  int c, p, d;
  int cmin, cmax;   // the columns of this warp
  __device__ __forceinline__ CtaPlace() {
    using C = CtaShape<LIMBS>;
    c = threadIdx.x / C::P;
    p = threadIdx.x % C::P;
    d = threadIdx.x;
    cmin = (threadIdx.x & ~31u) / C::P;
    cmax = cmin + 32 / C::P - 1;
  }
};

// Sums of this lane's halves: columns c and N + c of a product (and of those added to it).
struct CtaSums {
  uint64_t ll, lh, hl, hh;
};

enum CtaCols : int { kColsFull = 0, kColsLow = 1, kColsHigh = 2 };

// Adds x y's terms x_i y_j, i = p mod P, of columns i + j = c and N + c.  kColsLow: column c only.  kColsHigh:
// N + c, and c where the warp holds one of the three below N.
template <int LIMBS, int MODE>
__device__ __forceinline__ void cta_accumulate(CtaSums &a, const CtaPlace<LIMBS> &me, const double *x,
                                               const double *y) {
  using C = CtaShape<LIMBS>;
  const double *const xp = x + me.p, *const yp = y + C::N + me.c - me.p;
#pragma unroll
  for (int k0 = 0; k0 < C::K; k0 += C::CHUNK) {
    constexpr int L = C::CHUNK;
    if (C::CHUNK < C::K) {
      if (MODE == kColsLow && C::P * k0 > me.cmax) break;
      if (MODE == kColsHigh && C::P * (k0 + L) <= me.cmin + 1 && me.cmax < C::N - 3) continue;
    }
    double u[L], v[L], h[L], l[L];
#pragma unroll
    for (int k = 0; k < L; k++) {
      if (k0 + k >= C::K) continue;
      u[k] = xp[C::P * (k0 + k)];
      v[k] = yp[-C::P * (k0 + k)];
    }
#pragma unroll
    for (int k = 0; k < L; k++) {
      if (k0 + k >= C::K) continue;
      h[k] = __fma_rz(u[k], v[k], kDigHi);
    }
#pragma unroll
    for (int k = 0; k < L; k++) {
      if (k0 + k >= C::K) continue;
      l[k] = __fma_rz(u[k], v[k], __dsub_rn(kDigLo, h[k]));
    }
#pragma unroll
    for (int k = 0; k < L; k++) {
      if (k0 + k >= C::K) continue;
      const int i = me.p + C::P * (k0 + k);
      if (i <= me.c) {
        a.ll += dig_bits(l[k]);
        a.lh += dig_bits(h[k]);
      } else if (MODE != kColsLow && (C::N % C::P == 0 || i < C::N)) {
        a.hl += dig_bits(l[k]);
        a.hh += dig_bits(h[k]);
      }
    }
  }
}

// The groups' sums over their lanes, to s.low and s.high: each step halves the values a lane holds.
template <int LIMBS, bool BOTH>
__device__ __forceinline__ void cta_columns(CtaSmem<LIMBS> &s, const CtaPlace<LIMBS> &me, const CtaSums &a) {
  using C = CtaShape<LIMBS>;
  const bool odd = me.p & 1;
  uint64_t v = (odd ? a.lh : a.ll) + __shfl_xor_sync(kFull, odd ? a.ll : a.lh, 1);
  if (BOTH) {
    const uint64_t w = (odd ? a.hh : a.hl) + __shfl_xor_sync(kFull, odd ? a.hl : a.hh, 1);
    const bool up = me.p & 2;
    v = (up ? w : v) + __shfl_xor_sync(kFull, up ? v : w, 2);
  } else {
    v += __shfl_xor_sync(kFull, v, 2);
  }
  if (C::P == 8) v += __shfl_xor_sync(kFull, v, 4);
  if (me.p < (BOTH ? 4 : 2) && me.c < C::N) (odd ? s.high : s.low)[2 + (me.p & 2 ? C::N : 0) + me.c] = v;
  __syncthreads();
}

// Column j, -1 <= j < 2 N, of one product (of `products`) as a true signed sum.
template <int LIMBS>
__device__ __forceinline__ uint64_t cta_column(const CtaSmem<LIMBS> &s, int j, uint32_t products) {
  constexpr int N = CtaShape<LIMBS>::N;
  const int pairs = j < N ? j + 1 : 2 * N - 1 - j, below = j < 1 ? 0 : j - 1 < N ? j : 2 * N - j;
  return s.low[2 + j] + s.high[1 + j] -
         products * ((uint64_t)pairs * kDigLoBits64 + (uint64_t)below * kDigHiBits64);
}

// The digit of a column: its balanced low 52 bits and the carry of the column below.
__device__ __forceinline__ double cta_digit(uint64_t v, uint64_t below) {
  const uint32_t u = (uint32_t)(v >> 32) + 0x80080000u, b = (uint32_t)(below >> 32) + 0x80080000u;  // as dig_settle
  const double r = __dsub_rn(__hiloint2double((int)((u & 0xfffffu) | 0x43300000u), (int)(uint32_t)v),
                             0x1p53 + 0x1p51 + 2048.0);
  return __dadd_rn(r, __hiloint2double(0x43300000, (int)(b >> 20)));
}

// Stores digit d of an operand; role y: twice.
template <int LIMBS>
__device__ __forceinline__ void cta_put(double *v, int d, double x, bool twice) {
  v[d] = x;
  if (twice) v[CtaShape<LIMBS>::N + d] = x;
}

// out = the low columns of s (+ add at digit 0) mod R.
template <int LIMBS>
__device__ __forceinline__ void cta_low_digits(CtaSmem<LIMBS> &s, const CtaPlace<LIMBS> &me, double *out, bool twice,
                                               uint32_t add = 0) {
  if (me.d < CtaShape<LIMBS>::N) {
    const uint64_t v = cta_column(s, me.d, 1), below = cta_column(s, me.d - 1, 1);
    cta_put<LIMBS>(out, me.d, cta_digit(v + (me.d == 0 ? add : 0u), me.d == 0 ? 0 : below + (me.d == 1 ? add : 0u)),
                   twice);
  }
  __syncthreads();
}

// out = x y mod R (+ add at digit 0); y of role y.  out may alias x or y.
template <int LIMBS>
__device__ __forceinline__ void cta_low_product(CtaSmem<LIMBS> &s, const CtaPlace<LIMBS> &me, double *out, bool twice,
                                                const double *x, const double *y, uint32_t add = 0) {
  CtaSums a = {0, 0, 0, 0};
  cta_accumulate<LIMBS, kColsLow>(a, me, x, y);
  cta_columns<LIMBS, false>(s, me, a);
  cta_low_digits(s, me, out, twice, add);
}

// r = a b R^-1 mod N (|r| <= N); b of role y, r too if `twice`.  r may alias a or b.
template <int LIMBS>
__device__ __forceinline__ void mont_cta(CtaSmem<LIMBS> &s, const CtaPlace<LIMBS> &me, double *r, bool twice,
                                         const double *a, const double *b) {
  constexpr int N = CtaShape<LIMBS>::N;
  CtaSums u = {0, 0, 0, 0};
  cta_accumulate<LIMBS, kColsFull>(u, me, a, b);
  cta_columns<LIMBS, false>(s, me, u);
  cta_low_digits(s, me, s.t, false);
  cta_low_product(s, me, s.m, false, s.t, s.np);
  cta_accumulate<LIMBS, kColsHigh>(u, me, s.m, s.n);
  cta_columns<LIMBS, true>(s, me, u);
  if (me.d < N) {
    // c = the low half / R: column N - 1 with what column N - 2 carries into it
    const uint64_t v = cta_column(s, N + me.d, 2), v1 = cta_column(s, N + me.d - 1, 2),
                   v2 = cta_column(s, N + me.d - 2, 2);
    cta_put<LIMBS>(r, me.d, cta_digit(v, me.d == 0 ? v1 + (uint64_t)((int64_t)v2 >> 52) : v1), twice);
  }
  __syncthreads();
}

// Digit p of the number with limbs limb(j), balanced (as dig_from_limbs).
template <class Limb>
__device__ __forceinline__ double cta_limb_digit(Limb limb, uint32_t p) {
  const uint32_t o = 52 * p, w = o >> 5, sh = o & 31;
  uint64_t v = ((uint64_t)limb(w + 1) << 32 | limb(w)) >> sh;
  if (sh) v |= (uint64_t)limb(w + 2) << (64 - sh);
  v &= kDigMask;
  const uint32_t below = o ? (limb((o - 1) >> 5) >> ((o - 1) & 31)) & 1u : 0u;
  return (double)((int64_t)v - (int64_t)((v >> 51) << 52) + (int64_t)below);
}

// s.np = -N^-1 mod R by Newton's iteration y <- y (2 + N y), which doubles the correct low digits of y.
template <int LIMBS>
__device__ __forceinline__ void cta_neg_inverse(CtaSmem<LIMBS> &s, const CtaPlace<LIMBS> &me, uint64_t inv) {
  constexpr int N = CtaShape<LIMBS>::N;
  const auto limb = [&](uint32_t j) { return j == 0 ? (uint32_t)inv : j == 1 ? (uint32_t)(inv >> 32) & 0xfffffu : 0u; };
  if (threadIdx.x < N) cta_put<LIMBS>(s.np, me.d, me.d ? 0.0 : cta_limb_digit(limb, 0), true);
  __syncthreads();
#pragma unroll 1
  for (int digits = 1; digits < N; digits *= 2) {
    cta_low_product(s, me, s.m, false, s.n, s.np, 2);
    cta_low_product(s, me, s.np, true, s.m, s.np);
  }
}

// acc = R^2 mod N: warp 0 doubles 2^(bitlen N - 1) exactly on limbs up to 2^(52 N + e), 52 N = e 2^j with e odd
// (Montgomery form of 2^e), then j Montgomery squarings.  N = 1 gives 0.
template <int LIMBS>
__device__ __forceinline__ void cta_r2(CtaSmem<LIMBS> &s, const CtaPlace<LIMBS> &me, const PowmArgs &a, uint32_t em) {
  constexpr int N = CtaShape<LIMBS>::N, L = LIMBS / 32;
  constexpr uint32_t bits = 52u * N, j = N == 40 ? 5 : N == 80 ? 6 : 4, e = bits >> j;
  static_assert(bits == e << j && e % 2 == 1, "52 N = e 2^j");
  uint32_t *const limbs = reinterpret_cast<uint32_t *>(s.t);
  if (threadIdx.x < 32) {
    Group<32> G;
    uint32_t n[L], v[L];
    load_lane_limbs<32, L>(n, a.mod.limbs, a.mod.nlimbs, a.mod.stride, em, G.lane);
    const uint32_t b = dbitlen<32, L>(G, n);
    const uint32_t tb = b > 1 ? b - 1 : 0;
#pragma unroll
    for (int k = 0; k < L; k++) v[k] = b > 1 && (G.lane * L + k) == (tb >> 5) ? 1u << (tb & 31) : 0u;
    const uint32_t doublings = b > 1 ? bits + e - tb : 0;
#pragma unroll 1
    for (uint32_t d = 0; d < doublings; d++) dmod_double<32, L>(G, v, n, true);
#pragma unroll
    for (int k = 0; k < L; k++) limbs[G.lane * L + k] = v[k];
  }
  __syncthreads();
  if (threadIdx.x < N)
    cta_put<LIMBS>(s.acc, me.d,
                   cta_limb_digit([&](uint32_t q) { return q < (uint32_t)LIMBS ? limbs[q] : 0u; }, me.d), true);
  __syncthreads();
#pragma unroll 1
  for (uint32_t q = 0; q < j; q++) mont_cta(s, me, s.acc, true, s.acc, s.acc);
}

// Copies N digits within shared memory, to an operand of role y (every thread calls it).
template <int LIMBS>
__device__ __forceinline__ void cta_copy(double *dst, const double *src) {
  if (threadIdx.x < CtaShape<LIMBS>::N) cta_put<LIMBS>(dst, threadIdx.x, src[threadIdx.x], true);
  __syncthreads();
}

// One exponentiation per CTA.  Sliding window over the exponent's own bits
// (public exponents), or CT: the fixed window over the exponent's whole
// precision (the same schedule for every exponent).  The window table
// (sliding: slot 0 = Mont(1), slot j = Mont(x^(2j - 1)); fixed: slot e =
// Mont(x^e)) is in shared memory after the CtaSmem block.
template <int LIMBS, bool CT>
__global__ void __launch_bounds__(CtaShape<LIMBS>::THREADS, 1) powm_cta_kernel(PowmArgs a) {
  using C = CtaShape<LIMBS>;
  constexpr int N = C::N;
  extern __shared__ uint4 cta_dyn_smem[];
  CtaSmem<LIMBS> &s = *reinterpret_cast<CtaSmem<LIMBS> *>(cta_dyn_smem);
  double *table = reinterpret_cast<double *>(reinterpret_cast<char *>(cta_dyn_smem) + sizeof(CtaSmem<LIMBS>));
  const CtaPlace<LIMBS> me;
  const uint32_t inst = a.start + blockIdx.x;
  const uint32_t i = threadIdx.x;
  const uint32_t eb = in_element(a.base, inst), ee = in_element(a.exp, inst), em = in_element(a.mod, inst);
  const auto mod_limb = [&](uint32_t j) { return load_limb(a.mod.limbs, a.mod.nlimbs, a.mod.stride, em, j); };
  for (uint32_t w = i; w < sizeof(CtaSmem<LIMBS>) / 8; w += C::THREADS) reinterpret_cast<uint64_t *>(&s)[w] = 0;
  __syncthreads();
  if (i < N) {
    cta_put<LIMBS>(s.n, i, cta_limb_digit(mod_limb, i), true);
    cta_put<LIMBS>(
        s.x, i,
        cta_limb_digit([&](uint32_t j) { return load_limb(a.base.limbs, a.base.nlimbs, a.base.stride, eb, j); }, i),
        true);
    s.one[i] = i == 0 ? 1.0 : 0.0;
  }
  __syncthreads();
  // x may be >= N (any base below R / 4): x mod N comes out of Mont(x, R^2) = x R mod N
  cta_neg_inverse(s, me, dig_neg_inv(mod_limb(0), mod_limb(1)));
  cta_r2(s, me, a, em);
  const uint32_t W = a.window;
  const bool sliding = !CT;
  // table
  double *t1 = table + N;
  mont_cta(s, me, t1, false, s.x, s.acc);       // Mont(x)
  mont_cta(s, me, table, false, s.one, s.acc);  // Mont(1) = R mod N
  cta_copy<LIMBS>(s.x, t1);
  if (sliding) {
    mont_cta(s, me, s.x, true, t1, s.x);  // Mont(x^2)
#pragma unroll 1
    for (uint32_t j = 2; j <= (1u << (W - 1)); j++) mont_cta(s, me, table + j * N, false, table + (j - 1) * N, s.x);
  } else {
#pragma unroll 1
    for (uint32_t j = 2; j < (1u << W); j++) mont_cta(s, me, table + j * N, false, table + (j - 1) * N, s.x);
  }
  if (sliding) {
    // scan from the exponent's top bit
    int32_t top = -1;
    for (int32_t j = (int32_t)a.exp.nlimbs - 1; j >= 0; j--) {
      const uint32_t v = load_limb(a.exp.limbs, a.exp.nlimbs, a.exp.stride, ee, (uint32_t)j);
      if (v) {
        top = j * 32 + 31 - (int32_t)__clz(v);
        break;
      }
    }
    cta_copy<LIMBS>(s.acc, table);  // Mont(1)
    ExpCursor cur;
    cursor_init(cur, a.exp, ee, top);
    uint32_t sq, idx;
    bool first = true;
    while (true) {
      const bool more = next_window(a.exp, ee, cur, W, &sq, &idx);
      if (first && more) {
        // the accumulator is Mont(1): skip the squarings and take the first window's entry
        cta_copy<LIMBS>(s.acc, table + idx * N);
        first = false;
        continue;
      }
      // sq squarings and, unless the exponent ends, the window's entry: one product in the code
#pragma unroll 1
      for (uint32_t q = 0; q < sq + (more ? 1u : 0u); q++)
        mont_cta(s, me, s.acc, true, q < sq ? s.acc : table + idx * N, s.acc);
      if (!more) break;
    }
  } else {
    const uint32_t nwin = (a.exp.nlimbs * 32 + W - 1) / W;
    cta_copy<LIMBS>(s.acc, table + exp_window(a.exp, ee, (nwin - 1) * W, W) * N);
#pragma unroll 1
    for (int32_t wi = (int32_t)nwin - 2; wi >= 0; wi--) {
      const uint32_t win = exp_window(a.exp, ee, (uint32_t)wi * W, W);
#pragma unroll 1
      for (uint32_t q = 0; q <= W; q++) mont_cta(s, me, s.acc, true, q < W ? s.acc : table + win * N, s.acc);
    }
  }
  mont_cta(s, me, s.acc, false, s.one, s.acc);
  // into [0, N) on warp 0, then to limbs
  constexpr int D = (N + 31) / 32;
  uint64_t *const st = reinterpret_cast<uint64_t *>(s.t);
  if (i < 32) {
    Group<32> G;
    double v[D], n[D];
#pragma unroll
    for (int k = 0; k < D; k++) {
      const uint32_t p = G.lane * D + k;
      v[k] = p < N ? s.acc[p] : 0.0;
      n[k] = p < N ? s.n[p] : 0.0;
    }
    int64_t c[D];
    dig_canon<32, D>(G, c, v, n);
#pragma unroll
    for (int k = 0; k < D; k++)
      if (G.lane * D + k < N) st[G.lane * D + k] = (uint64_t)c[k];
  }
  __syncthreads();
  const uint32_t o = out_element(a.out, inst);
  if (o < a.out.count)
    for (uint32_t g = i; g < div_up(a.out.nlimbs, 4); g += C::THREADS)
      store_group(a.out.limbs, a.out.nlimbs, a.out.stride, o, g, dig_group(st, N, g));
}

}  // namespace xmpb

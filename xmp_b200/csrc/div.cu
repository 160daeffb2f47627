// xmpIntegersDiv/Mod/DivMod[Async] (replaces src/div.cu:26-517 and the
// kernels regmp_/digitmp_div/mod/divmod_kernel, implementations.h:436-763,
// with RegMP div_rem/rem (regmp/div.h:397-686) and DigitMP div
// (digitmp/div.h:109-526)).
//
// q = floor(a / b), r = a mod b.  Division by zero leaves q = a and r = 0
// (the reference's RegMP behaviour, regmp/div.h:594-596).
//
// Algorithm: schoolbook long division (Knuth, TAOCP vol. 2, 4.3.1, algorithm
// D).  The divisor is normalised by S = 32z + s bits so that its top limb has
// its top bit set (z whole limbs, s bits); the normalised divisor lives in
// registers (BN limbs, a compile-time class) together with a BN+1 limb window
// of the partial remainder.  The shifted dividend is never materialised: each
// step pulls its next limb straight from the interleaved input with the
// funnel shift applied.  The quotient digit estimate divides the top three
// window limbs by the top two divisor limbs with a precomputed reciprocal
// (Moller & Granlund, "Improved division by invariant integers", IEEE TC
// 2011, algorithm 5; one-limb divisors and the scratch kernel: algorithm 4,
// two limbs by one, refined against the second divisor limb); the
// multiply-subtract then needs at most one add-back.
// Larger divisors (up to 512 limbs) spread divisor and window over the lanes of
// a group; beyond that the same algorithm keeps them in the scratch arena.
#include "internal.h"
#include "carry.cuh"
#include "lanes.cuh"
#include "tune.h"
#include <algorithm>

using namespace xmpb;

namespace xmpb {

struct DivArgs {
  ArrayView a, b;
  OutView q, r;  // q.limbs or r.limbs may be null (Mod / Div)
  uint32_t count;
  uint32_t *scratch;  // large path: (2*nb + 1) words per thread, interleaved
  uint32_t T;
};

// floor((2^64 - 1) / d) - 2^32 for normalised d (top bit set).
__device__ __forceinline__ uint32_t reciprocal_2by1(uint32_t d) {
  return (uint32_t)(0xffffffffffffffffull / d - 0x100000000ull);
}

// (u1:u0) / d with u1 < d, d normalised, v = reciprocal_2by1(d).
__device__ __forceinline__ uint32_t div_2by1(uint32_t u1, uint32_t u0, uint32_t d, uint32_t v, uint32_t *rem) {
  uint64_t q = (uint64_t)v * u1;
  q += ((uint64_t)(u1 + 1) << 32) | u0;
  uint32_t q1 = (uint32_t)(q >> 32), q0 = (uint32_t)q;
  uint32_t r = u0 - q1 * d;
  if (r > q0) {
    q1--;
    r += d;
  }
  if (r >= d) {
    q1++;
    r -= d;
  }
  *rem = r;
  return q1;
}

// Quotient digit estimate from the window top (w2:w1:w0) and divisor top (d1:d0):
// floor((w2:w1)/d1) refined with w0 and d0; at most one too large.
__device__ __forceinline__ uint32_t estimate_q(uint32_t w2, uint32_t w1, uint32_t w0, uint32_t d1, uint32_t d0,
                                               uint32_t v, bool have_d0) {
  uint32_t qhat, rhat;
  bool rhat_big = false;
  if (w2 >= d1) {
    qhat = 0xffffffffu;
    uint64_t rr = (uint64_t)w1 + d1;  // (w2:w1) - qhat*d1 with w2 == d1
    rhat = (uint32_t)rr;
    rhat_big = (rr >> 32) != 0;
  } else {
    qhat = div_2by1(w2, w1, d1, v, &rhat);
  }
  if (have_d0) {
    for (int it = 0; it < 2 && !rhat_big; it++) {
      uint64_t lhs = (uint64_t)qhat * d0;
      uint64_t rhs = ((uint64_t)rhat << 32) | w0;
      if (lhs <= rhs) break;
      qhat--;
      uint64_t rr = (uint64_t)rhat + d1;
      rhat = (uint32_t)rr;
      rhat_big = (rr >> 32) != 0;
    }
  }
  return qhat;
}

// Reciprocal of the normalised two-limb divisor (d1:d0) for div_3by2: floor((2^96 - 1) / (d1:d0)) - 2^32
// (Moller & Granlund 2011, algorithm 6, from the one-limb reciprocal).
__device__ __forceinline__ uint32_t reciprocal_3by2(uint32_t d1, uint32_t d0) {
  uint32_t v = reciprocal_2by1(d1);
  uint32_t p = d1 * v + d0;
  if (p < d0) {
    v--;
    if (p >= d1) {
      v--;
      p -= d1;
    }
    p -= d1;
  }
  const uint64_t t = (uint64_t)v * d0;
  const uint32_t t1 = (uint32_t)(t >> 32);
  p += t1;
  if (p < t1) {
    v--;
    if (((uint64_t)p << 32 | (uint32_t)t) >= ((uint64_t)d1 << 32 | d0)) v--;
  }
  return v;
}

// Quotient digit estimate: floor((w2:w1:w0) / (d1:d0)) for (w2:w1) <= (d1:d0), at most one too large for the
// whole divisor (algorithm 5 of the same paper: one wide multiply by the reciprocal and two corrections
// without branches, where a digit over d1 alone needs up to four branches to reach the same estimate).
__device__ __forceinline__ uint32_t div_3by2(uint32_t w2, uint32_t w1, uint32_t w0, uint32_t d1, uint32_t d0,
                                             uint32_t v) {
  const uint64_t D = (uint64_t)d1 << 32 | d0;
  const uint64_t u = (uint64_t)w2 << 32 | w1;
  const uint64_t q = (uint64_t)v * w2 + u;
  uint32_t q1 = (uint32_t)(q >> 32);
  uint64_t r = ((uint64_t)(w1 - q1 * d1) << 32 | w0) - (uint64_t)d0 * q1 - D;
  q1++;
  if ((uint32_t)(r >> 32) >= (uint32_t)q) {
    q1--;
    r += D;
  }
  if (r >= D) q1++;
  return u >= D ? 0xffffffffu : q1;
}

struct ShiftedDividend {
  const ArrayView *a;
  uint32_t e;
  int32_t z;
  uint32_t s;
  // limb t of a * 2^(32z + s)
  __device__ __forceinline__ uint32_t operator()(int32_t t) const {
    int32_t j = t - z;
    uint32_t hi = (j >= 0 && j < (int32_t)a->nlimbs) ? load_limb(a->limbs, a->nlimbs, a->stride, e, (uint32_t)j) : 0u;
    if (s == 0) return hi;
    uint32_t lo = (j - 1 >= 0 && j - 1 < (int32_t)a->nlimbs) ? load_limb(a->limbs, a->nlimbs, a->stride, e, (uint32_t)(j - 1)) : 0u;
    return (hi << s) | (lo >> (32 - s));
  }
};

// Limbs of one instance read through a one-group cache: walking the limbs up
// or down loads each 128-bit group once instead of one 4-byte word per limb.
struct LimbCursor {
  const ArrayView *a;
  uint32_t e;
  int32_t g;
  uint4 v;
  __device__ __forceinline__ uint32_t operator()(int32_t j) {
    if (j < 0 || j >= (int32_t)a->nlimbs) return 0u;
    const int32_t gg = j >> 2;
    if (gg != g) {
      v = load_group(a->limbs, a->nlimbs, a->stride, e, (uint32_t)gg);
      g = gg;
    }
    const uint32_t r = j & 3;
    return r == 0 ? v.x : r == 1 ? v.y : r == 2 ? v.z : v.w;
  }
};

// limb t of a * 2^(32z + s), through two cursors (the limb and the one below it)
struct ShiftedCursor {
  LimbCursor hi, lo;
  int32_t z;
  uint32_t s;
  __device__ __forceinline__ uint32_t operator()(int32_t t) {
    const int32_t j = t - z;
    const uint32_t h = hi(j);
    if (s == 0) return h;
    return (h << s) | (lo(j - 1) >> (32 - s));
  }
};

__device__ __forceinline__ void write_limb(const OutView &o, uint32_t e, uint32_t j, uint32_t v) {
  if (j < o.nlimbs) limb_ref(o.limbs, o.stride, e, j) = v;
}
__device__ __forceinline__ void zero_limbs(const OutView &o, uint32_t e, uint32_t from) {
  for (uint32_t j = from; j < o.nlimbs; j++) limb_ref(o.limbs, o.stride, e, j) = 0;
}

// Special cases shared by both paths; returns true when the instance is done.
__device__ __forceinline__ bool div_trivial(const DivArgs &d, uint32_t ea, uint32_t eqo, uint32_t ero, int32_t bt,
                                            int32_t m) {
  if (bt < 0) {  // divisor 0: q = a, r = 0
    if (d.q.limbs) {
      for (uint32_t j = 0; j < d.q.nlimbs; j++)
        limb_ref(d.q.limbs, d.q.stride, eqo, j) = load_limb(d.a.limbs, d.a.nlimbs, d.a.stride, ea, j);
    }
    if (d.r.limbs) zero_limbs(d.r, ero, 0);
    return true;
  }
  if (m < 0) {  // a has fewer limbs than b: q = 0, r = a
    if (d.q.limbs) zero_limbs(d.q, eqo, 0);
    if (d.r.limbs) {
      for (uint32_t j = 0; j < d.r.nlimbs; j++)
        limb_ref(d.r.limbs, d.r.stride, ero, j) = load_limb(d.a.limbs, d.a.nlimbs, d.a.stride, ea, j);
    }
    return true;
  }
  return false;
}

template <int BN>
__global__ void __launch_bounds__(256) divmod_reg_kernel(DivArgs d) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.count) return;
  const uint32_t ea = in_element(d.a, i), eb = in_element(d.b, i);
  const uint32_t eqo = d.q.limbs ? out_element(d.q, i) : 0, ero = d.r.limbs ? out_element(d.r, i) : 0;
  if ((d.q.limbs && eqo >= d.q.count) || (d.r.limbs && ero >= d.r.count)) return;

  // Top nonzero divisor limb.
  int32_t bt = -1;
  for (int32_t j = (int32_t)d.b.nlimbs - 1; j >= 0; j--)
    if (load_limb(d.b.limbs, d.b.nlimbs, d.b.stride, eb, j)) {
      bt = j;
      break;
    }
  const int32_t m = (int32_t)d.a.nlimbs - bt - 1;  // quotient limbs - 1
  if (div_trivial(d, ea, eqo, ero, bt, m)) return;

  const int32_t z = BN - 1 - bt;
  const uint32_t s = __clz(load_limb(d.b.limbs, d.b.nlimbs, d.b.stride, eb, bt));
  uint32_t V[BN];
  {
    ShiftedDividend sb{&d.b, eb, z, s};
#pragma unroll
    for (int k = 0; k < BN; k++) V[k] = sb(k);
  }
  uint32_t W[BN + 1];
  // The digit of the present window: estimate, W -= qh * V (one mul.wide per limb; low halves at limbs 0 ..
  // BN - 1, high halves at 1 .. BN), one add-back at most.
  const uint32_t d1 = V[BN - 1], d0 = BN >= 2 ? V[BN >= 2 ? BN - 2 : 0] : 0u;
  const uint32_t v = BN >= 2 ? reciprocal_3by2(d1, d0) : reciprocal_2by1(d1);
  auto digit = [&]() -> uint32_t {
    uint32_t qh = BN >= 2 ? div_3by2(W[BN], W[BN - 1], W[BN >= 2 ? BN - 2 : 0], d1, d0, v)
                          : estimate_q(W[BN], W[BN - 1], 0u, d1, 0u, v, false);
    uint64_t p[BN];
#pragma unroll
    for (int k = 0; k < BN; k++) p[k] = mul_wide(qh, V[k]);
    W[0] = sub_cc(W[0], (uint32_t)p[0]);
#pragma unroll
    for (int k = 1; k < BN; k++) W[k] = subc_cc(W[k], (uint32_t)p[k]);
    W[BN] = subc(W[BN], 0u);
    W[1] = sub_cc(W[1], (uint32_t)(p[0] >> 32));
#pragma unroll
    for (int k = 2; k <= BN; k++) W[k] = subc_cc(W[k], (uint32_t)(p[k - 1] >> 32));
    if (W[BN] != 0) {  // estimate was one too large: add back
      qh--;
      W[0] = add_cc(W[0], V[0]);
#pragma unroll
      for (int k = 1; k < BN; k++) W[k] = addc_cc(W[k], V[k]);
      W[BN] = addc(W[BN], 0u);
    }
    return qh;
  };
  auto shift_in = [&](uint32_t limb) {
#pragma unroll
    for (int k = BN; k > 0; k--) W[k] = W[k - 1];
    W[0] = limb;
  };
  // quotient limbs collect in a group buffer and are stored 128 bits at a time
  uint32_t qb0 = 0, qb1 = 0, qb2 = 0, qb3 = 0;
  auto store_q = [&](uint32_t g) {
    if (d.q.limbs && g * 4 < d.q.nlimbs)
      store_group(d.q.limbs, d.q.nlimbs, d.q.stride, eqo, g, make_uint4(qb0, qb1, qb2, qb3));
  };
  if (z == 0) {
    // A divisor of the class's length, its usual case: the dividend's limbs come group by group, the next
    // one loaded ahead, and every digit knows its place in its group.  Against a cursor per limb (bounds, group
    // and component tests for two limbs a digit) and the branching digit estimate, dividends twice the
    // divisor's length: 512 bits x 262,144 63 -> 40.5 us, 1024 bits x 65,536 48 -> 30, 1536 bits x 32,768 57 ->
    // 34.  The quotient digits' chain bounds it, 512 bits x 262,144 move at 2.9 TB/s.
    {
      uint32_t hi = 0;
#pragma unroll
      for (int k = BN; k >= 0; k--) {
        const uint32_t lo = m + k > 0 ? load_limb(d.a.limbs, d.a.nlimbs, d.a.stride, ea, (uint32_t)(m + k - 1)) : 0u;
        if (k < BN) W[k] = __funnelshift_l(lo, hi, s);
        else W[k] = s ? lo >> (32 - s) : 0u;
        hi = lo;
      }
    }
    const int32_t top = (m - 1) >> 2;
    uint4 cur = m > 0 ? load_group(d.a.limbs, d.a.nlimbs, d.a.stride, ea, (uint32_t)top) : make_uint4(0, 0, 0, 0);
    int32_t skip = 3 - ((m - 1) & 3);  // places of the first group above the window
#pragma unroll 1
    for (int32_t g = top; g >= 0 && m > 0; g--) {
      const uint4 next = g > 0 ? load_group(d.a.limbs, d.a.nlimbs, d.a.stride, ea, (uint32_t)(g - 1))
                               : make_uint4(0, 0, 0, 0);
      if (skip < 1) {
        qb0 = digit();
        store_q((uint32_t)g + 1);
        qb1 = qb2 = qb3 = 0;
        shift_in(__funnelshift_l(cur.z, cur.w, s));
      }
      if (skip < 2) {
        qb3 = digit();
        shift_in(__funnelshift_l(cur.y, cur.z, s));
      }
      if (skip < 3) {
        qb2 = digit();
        shift_in(__funnelshift_l(cur.x, cur.y, s));
      }
      qb1 = digit();
      shift_in(__funnelshift_l(next.w, cur.x, s));
      cur = next;
      skip = 0;
    }
    qb0 = digit();
    store_q(0);
  } else {
    ShiftedCursor sa{LimbCursor{&d.a, ea, -1, make_uint4(0, 0, 0, 0)},
                     LimbCursor{&d.a, ea, -1, make_uint4(0, 0, 0, 0)}, z, s};
#pragma unroll
    for (int k = 0; k <= BN; k++) W[k] = sa(m + k);
    for (int32_t j = m; j >= 0; j--) {
      const uint32_t qh = digit();
      const uint32_t r4 = (uint32_t)j & 3u;
      qb0 = r4 == 0 ? qh : qb0;
      qb1 = r4 == 1 ? qh : qb1;
      qb2 = r4 == 2 ? qh : qb2;
      qb3 = r4 == 3 ? qh : qb3;
      if (r4 == 0) {
        store_q((uint32_t)j >> 2);
        qb0 = qb1 = qb2 = qb3 = 0;
      }
      if (j > 0) shift_in(sa(j - 1));
    }
  }
  // limbs above the quotient's top group
  if (d.q.limbs) zero_limbs(d.q, eqo, (uint32_t)(m / 4 + 1) * 4);
  if (d.r.limbs) {
    // remainder = W >> S
    if (z == 0) {
      const uint32_t rg = div_up(d.r.nlimbs, 4);
#pragma unroll
      for (int g = 0; g < (BN + 3) / 4; g++) {
        uint32_t o[4];
#pragma unroll
        for (int t = 0; t < 4; t++) {
          const int k = 4 * g + t;
          const uint32_t lo = k < BN ? W[k < BN ? k : 0] : 0u;
          const uint32_t hi = (k + 1 < BN) ? W[k + 1 < BN ? k + 1 : 0] : 0u;
          o[t] = s ? ((lo >> s) | (hi << (32 - s))) : lo;
        }
        if ((uint32_t)g < rg) store_group(d.r.limbs, d.r.nlimbs, d.r.stride, ero, g, make_uint4(o[0], o[1], o[2], o[3]));
      }
      for (uint32_t g = (BN + 3) / 4; g < rg; g++)
        store_group(d.r.limbs, d.r.nlimbs, d.r.stride, ero, g, make_uint4(0, 0, 0, 0));
    } else {
#pragma unroll
      for (int k = 0; k < BN; k++) {
        int32_t dst = k - z;
        if (dst >= 0) {
          uint32_t hi = (k + 1 < BN) ? W[k + 1 < BN ? k + 1 : 0] : 0u;
          uint32_t val = s ? ((W[k] >> s) | (hi << (32 - s))) : W[k];
          write_limb(d.r, ero, (uint32_t)dst, val);
        }
      }
      zero_limbs(d.r, ero, (uint32_t)(BN - z));
    }
  }
}

// Divisor and window over TPI lanes x L limbs (N = TPI * L >= divisor limbs), the word above the window
// (`top`) in every lane.  Every instance of a warp runs the quotient digits from the warp's highest down:
// above its own highest its window is below the divisor and the digit comes out 0.  A digit: estimate from
// the top lane's words (every lane computes it), each lane subtracts qh * V from its limbs, the lanes'
// borrow words go one lane up, and a ballot lookahead settles what is left of them (mont.cuh).  The chain
// from digit to digit is the bound (2048 / 1024 bits x 64 instances: 24 us against 31 us on one thread
// each); against the scratch kernel below: 4160 / 2080 bits x 10,001 456 -> 69 us, 8192 / 4096 x 4,096
// 1,617 -> 91 us, 16384 / 8192 x 2,048 5,533 -> 170 us.
template <int TPI, int L>
__global__ void __launch_bounds__(256) divmod_lanes_kernel(DivArgs d) {
  constexpr int N = TPI * L;
  Group<TPI> G;
  const uint64_t local = lane_instance<TPI>(blockIdx.x, blockDim.x, threadIdx.x);
  const bool valid = local < d.count;
  const uint32_t i = valid ? (uint32_t)local : d.count - 1;
  const uint32_t ea = in_element(d.a, i), eb = in_element(d.b, i);
  const uint32_t eqo = d.q.limbs ? out_element(d.q, i) : 0, ero = d.r.limbs ? out_element(d.r, i) : 0;
  const bool store = valid && !(d.q.limbs && eqo >= d.q.count) && !(d.r.limbs && ero >= d.r.count);

  uint32_t V[L];
  load_lane_limbs<TPI, L>(V, d.b.limbs, d.b.nlimbs, d.b.stride, eb, G.lane);
  const uint32_t bits = dbitlen<TPI, L>(G, V);
  const bool zero = bits == 0;  // division by zero: q = a, r = 0, written at the end
  const int32_t bt = zero ? N - 1 : (int32_t)(bits - 1) / 32;
  const int32_t z = N - 1 - bt;
  const uint32_t s = zero ? 0 : (32 - bits % 32) % 32;
  {
    ShiftedDividend sb{&d.b, eb, z, s};
#pragma unroll
    for (int k = 0; k < L; k++) V[k] = sb((int32_t)(G.lane * L) + k);
  }
  uint32_t d1 = G.bcast(V[L - 1], TPI - 1);
  const uint32_t d0 = G.bcast(V[L - 2], TPI - 1);
  if (zero) d1 = 0x80000000u;
  const uint32_t v = reciprocal_3by2(d1, d0);
  ShiftedCursor sa{LimbCursor{&d.a, ea, -1, make_uint4(0, 0, 0, 0)}, LimbCursor{&d.a, ea, -1, make_uint4(0, 0, 0, 0)},
                   z, s};
  const int32_t m = max(0, (int32_t)__reduce_max_sync(kFull, (uint32_t)max(0, (int32_t)d.a.nlimbs - bt - 1)));
  uint32_t W[L], top = sa(m + N);
#pragma unroll
  for (int k = L - 1; k >= 0; k--) W[k] = sa(m + (int32_t)(G.lane * L) + k);

  uint32_t qb0 = 0, qb1 = 0, qb2 = 0, qb3 = 0;
#pragma unroll 1
  for (int32_t j = m; j >= 0; j--) {
    uint32_t qh = div_3by2(top, G.bcast(W[L - 1], TPI - 1), G.bcast(W[L - 2], TPI - 1), d1, d0, v);
    const uint32_t next = j > 0 ? sa(j - 1) : 0u;
    uint64_t p[L];
    row_products<L>(p, V, qh);
    W[0] = sub_cc(W[0], (uint32_t)p[0]);
#pragma unroll
    for (int k = 1; k < L; k++) W[k] = subc_cc(W[k], (uint32_t)p[k]);
    uint32_t up = (uint32_t)(p[L - 1] >> 32) - subc(0u, 0u);
    W[1] = sub_cc(W[1], (uint32_t)(p[0] >> 32));
#pragma unroll
    for (int k = 2; k < L; k++) W[k] = subc_cc(W[k], (uint32_t)(p[k - 1] >> 32));
    up -= subc(0u, 0u);
    // the lanes' borrow words, then the one-bit borrows that these leave
    const uint32_t in = G.from_prev(up);
    W[0] = sub_cc(W[0], in);
#pragma unroll
    for (int k = 1; k < L; k++) W[k] = subc_cc(W[k], 0u);
    const uint32_t bo = 0u - subc(0u, 0u);
    uint32_t any = W[0];
#pragma unroll
    for (int k = 1; k < L; k++) any |= W[k];
    uint32_t out;
    const uint32_t bin = G.lookahead(bo, any == 0u, &out);
    W[0] = sub_cc(W[0], bin);
#pragma unroll
    for (int k = 1; k < L; k++) W[k] = subc_cc(W[k], 0u);
    top -= G.bcast(up, TPI - 1) + out;
    if (__any_sync(kFull, top != 0)) {  // an estimate was one too large: add the divisor back
      const uint32_t msk = top != 0 ? kFull : 0u;
      W[0] = add_cc(W[0], V[0] & msk);
#pragma unroll
      for (int k = 1; k < L; k++) W[k] = addc_cc(W[k], V[k] & msk);
      const uint32_t co = addc(0u, 0u);
      uint32_t ones = W[0];
#pragma unroll
      for (int k = 1; k < L; k++) ones &= W[k];
      const uint32_t ci = G.lookahead(co, ones == kFull, &out);
      W[0] = add_cc(W[0], ci);
#pragma unroll
      for (int k = 1; k < L; k++) W[k] = addc_cc(W[k], 0u);
      qh += msk;
    }
    const uint32_t r4 = (uint32_t)j & 3u;
    qb0 = r4 == 0 ? qh : qb0;
    qb1 = r4 == 1 ? qh : qb1;
    qb2 = r4 == 2 ? qh : qb2;
    qb3 = r4 == 3 ? qh : qb3;
    if (r4 == 0) {
      const uint32_t g = (uint32_t)j >> 2;
      if (G.lane == 0 && store && !zero && d.q.limbs && g * 4 < d.q.nlimbs)
        store_group(d.q.limbs, d.q.nlimbs, d.q.stride, eqo, g, make_uint4(qb0, qb1, qb2, qb3));
      qb0 = qb1 = qb2 = qb3 = 0;
    }
    if (j > 0) {
      top = G.bcast(W[L - 1], TPI - 1);
      const uint32_t below = G.lane == 0 ? next : 0u;
      const uint32_t prev = G.from_prev(W[L - 1]);
#pragma unroll
      for (int k = L - 1; k > 0; k--) W[k] = W[k - 1];
      W[0] = G.lane == 0 ? below : prev;
    }
  }
  // remainder = W >> (32 z + s)
  const uint32_t above = G.from_next(W[0]);
  if (!store) return;
  if (d.q.limbs) {
    for (uint32_t g = zero ? G.lane : (uint32_t)m / 4 + 1 + G.lane; g * 4 < d.q.nlimbs; g += TPI)
      store_group(d.q.limbs, d.q.nlimbs, d.q.stride, eqo, g,
                  zero ? load_group(d.a.limbs, d.a.nlimbs, d.a.stride, ea, g) : make_uint4(0, 0, 0, 0));
  }
  if (d.r.limbs) {
    uint32_t R[L];
#pragma unroll
    for (int k = 0; k < L; k++) {
      const uint32_t hi = k + 1 < L ? W[k + 1 < L ? k + 1 : 0] : above;
      R[k] = zero ? 0u : s ? (W[k] >> s) | (hi << (32 - s)) : W[k];
    }
    if (z == 0) {
      store_lane_limbs<TPI, L>(R, d.r.limbs, d.r.nlimbs, d.r.stride, ero, G.lane);
    } else {
#pragma unroll
      for (int k = 0; k < L; k++) {
        const int32_t dst = (int32_t)(G.lane * L) + k - z;
        if (dst >= 0) write_limb(d.r, ero, (uint32_t)dst, R[k]);
      }
    }
    for (uint32_t j = N - z + G.lane; j < d.r.nlimbs; j += TPI) limb_ref(d.r.limbs, d.r.stride, ero, j) = 0;
  }
}

// Same algorithm with the window and divisor in scratch (any divisor size).
__global__ void __launch_bounds__(256) divmod_stream_kernel(DivArgs d) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.count) return;
  const uint32_t ea = in_element(d.a, i), eb = in_element(d.b, i);
  const uint32_t eqo = d.q.limbs ? out_element(d.q, i) : 0, ero = d.r.limbs ? out_element(d.r, i) : 0;
  if ((d.q.limbs && eqo >= d.q.count) || (d.r.limbs && ero >= d.r.count)) return;
  int32_t bt = -1;
  for (int32_t j = (int32_t)d.b.nlimbs - 1; j >= 0; j--)
    if (load_limb(d.b.limbs, d.b.nlimbs, d.b.stride, eb, j)) {
      bt = j;
      break;
    }
  const int32_t m = (int32_t)d.a.nlimbs - bt - 1;
  if (div_trivial(d, ea, eqo, ero, bt, m)) return;
  const int32_t BN = bt + 1;  // exact divisor length: no whole-limb shift needed
  const uint32_t s = __clz(load_limb(d.b.limbs, d.b.nlimbs, d.b.stride, eb, bt));
  const size_t T = d.T;
  uint32_t *V = d.scratch + i;
  uint32_t *W = V + (size_t)d.b.nlimbs * T;
  ShiftedDividend sb{&d.b, eb, 0, s};
  for (int32_t k = 0; k < BN; k++) V[k * T] = sb(k);
  const uint32_t dtop = V[(BN - 1) * T], dnext = BN >= 2 ? V[(BN - 2) * T] : 0u;
  const uint32_t v = reciprocal_2by1(dtop);
  ShiftedDividend sa{&d.a, ea, 0, s};
  // W[k] for k = 0..BN holds window limb k; the window slides by moving its base.
  // Stored as a ring of BN+1 words: limb k at W[((base + k) % (BN+1)) * T].
  const int32_t WN = BN + 1;
  int32_t base = 0;
  auto wref = [&](int32_t k) -> uint32_t & { return W[(size_t)((base + k) % WN) * T]; };
  for (int32_t k = 0; k <= BN; k++) wref(k) = sa(m + k);
  for (int32_t j = m; j >= 0; j--) {
    uint32_t qh = estimate_q(wref(BN), wref(BN - 1), BN >= 2 ? wref(BN - 2) : 0u, dtop, dnext, v, BN >= 2);
    // W -= qh * V with a running borrow and product carry.
    uint32_t borrow = 0, carry = 0;
    for (int32_t k = 0; k < BN; k++) {
      uint64_t p = (uint64_t)qh * V[k * T] + carry;
      carry = (uint32_t)(p >> 32);
      uint64_t t = (uint64_t)wref(k) - (uint32_t)p - borrow;
      wref(k) = (uint32_t)t;
      borrow = (uint32_t)(t >> 63);
    }
    uint64_t t = (uint64_t)wref(BN) - carry - borrow;
    wref(BN) = (uint32_t)t;
    if ((uint32_t)t != 0) {
      qh--;
      uint32_t c = 0;
      for (int32_t k = 0; k < BN; k++) {
        uint64_t s2 = (uint64_t)wref(k) + V[k * T] + c;
        wref(k) = (uint32_t)s2;
        c = (uint32_t)(s2 >> 32);
      }
      wref(BN) += c;
    }
    if (d.q.limbs) write_limb(d.q, eqo, (uint32_t)j, qh);
    if (j > 0) {
      // slide: new limb k = old limb k-1, new limb 0 = next dividend limb
      base = (base + WN - 1) % WN;
      wref(0) = sa(j - 1);
    }
  }
  if (d.q.limbs) zero_limbs(d.q, eqo, (uint32_t)(m + 1));
  if (d.r.limbs) {
    for (int32_t k = 0; k < BN; k++) {
      uint32_t hi = (k + 1 < BN) ? wref(k + 1) : 0u;
      uint32_t val = s ? ((wref(k) >> s) | (hi << (32 - s))) : wref(k);
      write_limb(d.r, ero, (uint32_t)k, val);
    }
    zero_limbs(d.r, ero, (uint32_t)BN);
  }
}

typedef void (*DivLaunch)(const DivArgs &, int, cudaStream_t);
template <int BN>
static void launch_div(const DivArgs &d, int threads, cudaStream_t s) {
  divmod_reg_kernel<BN><<<grid_for(d.count, threads), threads, 0, s>>>(d);
}
static DivLaunch pick_div(uint32_t nb) {
  if (nb <= 1) return launch_div<1>;
  if (nb <= 2) return launch_div<2>;
  if (nb <= 4) return launch_div<4>;
  if (nb <= 6) return launch_div<6>;
  if (nb <= 8) return launch_div<8>;
  if (nb <= 12) return launch_div<12>;
  if (nb <= 16) return launch_div<16>;
  if (nb <= 24) return launch_div<24>;
  if (nb <= 32) return launch_div<32>;
  if (nb <= 48) return launch_div<48>;
  if (nb <= 64) return launch_div<64>;
  return nullptr;
}

template <int TPI, int L>
static void launch_div_lanes(const DivArgs &d, int threads, cudaStream_t s) {
  divmod_lanes_kernel<TPI, L><<<grid_for((uint64_t)d.count * TPI, threads), threads, 0, s>>>(d);
}
// Whether lanes beat one thread per instance for a divisor that a register kernel holds: while the batch is
// too small to give every scheduler a register warp or half of one, and the divisor long enough.  Measured,
// register / lane kernel: 2048-bit divisors x 2^12 78.6 / 41.8 us, 2^14 78.5 / 68.8, 2^16 189 / 237; 1024 bits
// x 2^12 31.8 / 25.6, 2^14 33.5 / 31.1, 2^16 49.7 / 70.1; 768 bits x 2^12 23.9 / 21.3, 2^14 24.7 / 25.5; 512
// bits x 2^12 17.3 / 16.7, 2^16 23.1 / 29.1.
static bool div_lanes_preferred(uint32_t nb, uint32_t count, uint32_t sm_count) {
  return nb > 16 && count <= sm_count * (nb > 32 ? 128u : 64u);
}

// Lane kernel for a divisor of nb limbs (null: above 512); `wide` as in the multiply's lane path.
static DivLaunch pick_div_lanes(uint32_t nb, uint32_t count, uint32_t sm_count) {
  const bool wide = (uint64_t)count * round_up(nb, 16) / 16 < (uint64_t)sm_count * 4 * 2 * 32;
  if (nb <= 16) return launch_div_lanes<2, 8>;
  if (nb <= 32) return wide ? launch_div_lanes<4, 8> : launch_div_lanes<2, 16>;
  if (nb <= 48) return launch_div_lanes<4, 12>;
  if (nb <= 64) return wide ? launch_div_lanes<8, 8> : launch_div_lanes<4, 16>;
  if (nb <= 96) return launch_div_lanes<8, 12>;
  if (nb <= 128) return wide ? launch_div_lanes<16, 8> : launch_div_lanes<8, 16>;
  if (nb <= 256) return wide ? launch_div_lanes<32, 8> : launch_div_lanes<16, 16>;
  if (nb <= 512) return launch_div_lanes<32, 16>;
  return nullptr;
}

bool div_has_register_kernel(uint32_t nb) { return pick_div(nb) != nullptr; }

static xmpError_t divmod_common(xmpHandle_t h, xmpIntegers_t q, xmpIntegers_t r, xmpIntegers_t a, xmpIntegers_t b,
                                uint32_t count, int qi, int ri, int ai, int bi, const ElemConfig *forced) {
  xmpExecutionPolicy_t pol = h->policy;
  DivArgs d;
  d.a = view_in(a, pol->indices[ai], pol->indices_count[ai]);
  d.b = view_in(b, pol->indices[bi], pol->indices_count[bi]);
  d.count = count;
  d.scratch = nullptr;
  d.T = 0;
  DivLaunch launch = pol->algorithm == xmpAlgorithmDigitMP ? nullptr : pick_div(b->nlimbs);
  if (pol->algorithm == xmpAlgorithmRegMP && !launch) return xmpErrorUnsupported;
  ElemConfig cfg;
  int source = 0;  // 1: a choice set for this very shape
  if (forced) {
    cfg = *forced;
  } else if (pol->algorithm == xmpAlgorithmDefault) {
    int slot = tuner_lookup(h, xmpTuneDivMod, b->precision, 0, count, &source);
    ElemConfig t;
    if (slot >= 0 && elem_candidate(xmpTuneDivMod, b->nlimbs, slot, &t)) cfg = t;
  }
  if (cfg.variant == 1) launch = nullptr;
  else if (!launch && forced) return xmpErrorUnsupported;
  if ((pol->algorithm == xmpAlgorithmDefault || pol->algorithm == xmpAlgorithmDistributedMP) &&
      (!launch || (!forced && source != 1 && div_lanes_preferred(b->nlimbs, count, h->sm_count)))) {
    if (DivLaunch lanes = pick_div_lanes(b->nlimbs, count, h->sm_count)) launch = lanes;
  }
  const int threads = cfg.threads;

  OutTarget tq, tr;
  xmpError_t e;
  // Outputs are written digit by digit while the dividend is still being read: stage any alias.
  size_t q_bytes = q ? q->bytes : 0;
  bool q_stage = q && (q == a || q == b), r_stage = r && (r == a || r == b);
  if (q_stage || r_stage) {
    // size the in-place arena once so staging the second output cannot move the first
    e = ensure_tmp_out(h, (q_stage ? q_bytes : 0) + (r_stage ? r->bytes : 0));
    if (e != xmpErrorSuccess) return e;
  }
  if (q) {
    e = begin_output(h, q, q == a || q == b, true, &tq, 0);
    if (e != xmpErrorSuccess) return e;
  }
  if (r) {
    e = begin_output(h, r, r == a || r == b, true, &tr, tq.staged ? q_bytes : 0);
    if (e != xmpErrorSuccess) return e;
  }

  d.q = q ? view_out(q, tq.limbs, qi >= 0 ? pol->indices[qi] : nullptr) : OutView{nullptr, 0, 0, 0, nullptr};
  d.r = r ? view_out(r, tr.limbs, ri >= 0 ? pol->indices[ri] : nullptr) : OutView{nullptr, 0, 0, 0, nullptr};
  if (launch) {
    launch(d, threads, h->stream);
  } else {
    d.T = round_up(count, 256);
    e = ensure_scratch(h, (size_t)(2 * b->nlimbs + 1) * d.T * 4);
    if (e != xmpErrorSuccess) return e;
    d.scratch = (uint32_t *)h->scratch;
    divmod_stream_kernel<<<grid_for(count, threads), threads, 0, h->stream>>>(d);
  }
  if (q) {
    e = end_output(h, q, tq);
    if (e != xmpErrorSuccess) return e;
  }
  if (r) {
    e = end_output(h, r, tr);
    if (e != xmpErrorSuccess) return e;
  }
  return check_cuda();
}

xmpError_t divmod_entry(xmpHandle_t h, xmpIntegers_t q, xmpIntegers_t r, xmpIntegers_t a, xmpIntegers_t b,
                        uint32_t count, const ElemConfig *forced) {
  if (!h || !q || !r || !a || !b) return xmpErrorInvalidParameter;
  int dev = h->device;
  if (q->device != dev || r->device != dev || a->device != dev || b->device != dev) return xmpErrorInvalidDevice;
  if (count == 0) return xmpErrorSuccess;
  DeviceGuard guard(dev);
  xmpExecutionPolicy_t p = h->policy;
  if (r->count < count || q->count < count) return xmpErrorInvalidCount;
  if (p->indices[0] && p->indices_count[0] < count) return xmpErrorInvalidCount;
  if (p->indices[1] && p->indices_count[1] < count) return xmpErrorInvalidCount;
  if (q->precision < a->precision || r->precision < b->precision) return xmpErrorInvalidPrecision;
  if (q == r) return xmpErrorInvalidParameter;
  return divmod_common(h, q, r, a, b, count, 0, 1, 2, 3, forced);
}

static xmpError_t sync_after(xmpHandle_t h, xmpError_t e) {
  if (e != xmpErrorSuccess) return e;
  DeviceGuard guard(h->device);
  cudaStreamSynchronize(h->stream);
  return check_cuda();
}

}  // namespace xmpb

extern "C" {

xmpError_t XMPAPI xmpIntegersDivAsync(xmpHandle_t h, xmpIntegers_t q, const xmpIntegers_t a, const xmpIntegers_t b,
                                       uint32_t count) {
  if (!h || !q || !a || !b) return xmpErrorInvalidParameter;
  if (q->device != h->device || a->device != h->device || b->device != h->device) return xmpErrorInvalidDevice;
  if (count == 0) return xmpErrorSuccess;
  DeviceGuard guard(h->device);
  xmpExecutionPolicy_t p = h->policy;
  if (q->count < count) return xmpErrorInvalidCount;
  if (p->indices[0] && p->indices_count[0] < count) return xmpErrorInvalidCount;
  if (q->precision < a->precision) return xmpErrorInvalidPrecision;
  return divmod_common(h, q, nullptr, a, b, count, 0, -1, 1, 2, nullptr);
}
xmpError_t XMPAPI xmpIntegersDiv(xmpHandle_t h, xmpIntegers_t q, const xmpIntegers_t a, const xmpIntegers_t b,
                                  uint32_t count) {
  return sync_after(h, xmpIntegersDivAsync(h, q, a, b, count));
}

xmpError_t XMPAPI xmpIntegersModAsync(xmpHandle_t h, xmpIntegers_t m, const xmpIntegers_t a, const xmpIntegers_t b,
                                       uint32_t count) {
  if (!h || !m || !a || !b) return xmpErrorInvalidParameter;
  if (m->device != h->device || a->device != h->device || b->device != h->device) return xmpErrorInvalidDevice;
  if (count == 0) return xmpErrorSuccess;
  DeviceGuard guard(h->device);
  xmpExecutionPolicy_t p = h->policy;
  if (m->count < count) return xmpErrorInvalidCount;
  if (p->indices[0] && p->indices_count[0] < count) return xmpErrorInvalidCount;
  if (m->precision < b->precision) return xmpErrorInvalidPrecision;
  return divmod_common(h, nullptr, m, a, b, count, -1, 0, 1, 2, nullptr);
}
xmpError_t XMPAPI xmpIntegersMod(xmpHandle_t h, xmpIntegers_t m, const xmpIntegers_t a, const xmpIntegers_t b,
                                  uint32_t count) {
  return sync_after(h, xmpIntegersModAsync(h, m, a, b, count));
}

xmpError_t XMPAPI xmpIntegersDivModAsync(xmpHandle_t h, xmpIntegers_t q, xmpIntegers_t m, const xmpIntegers_t a,
                                          const xmpIntegers_t b, uint32_t count) {
  return divmod_entry(h, q, m, a, b, count, nullptr);
}
xmpError_t XMPAPI xmpIntegersDivMod(xmpHandle_t h, xmpIntegers_t q, xmpIntegers_t m, const xmpIntegers_t a,
                                     const xmpIntegers_t b, uint32_t count) {
  return sync_after(h, xmpIntegersDivModAsync(h, q, m, a, b, count));
}

}  // extern "C"

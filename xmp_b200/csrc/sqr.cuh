// Squaring-specialised Montgomery product: r = a^2 R^-1 mod N, almost reduced
// (r < R), for the exponentiation's squarings on one lane (the reference's
// per-thread sqr, regmp/sqr_imad.h:25-78, used by its powm model
// powm/three_n.h).
//
// Separated operand scanning: the square T = a^2 is formed first with each
// cross product a_i a_j (i < j) computed once and doubled, then reduced by the
// same quotient rows as mont_mul (acc += N q, shift one word) with the words
// of T fed into the accumulator as the rows reach them.  A 2n-limb square
// costs n(n+1)/2 products instead of n^2, so a Montgomery squaring costs about
// 3n^2/2 + n products instead of 2n^2 + n.
//
// T is formed in registers; the reduction takes T's low half as the
// accumulator and shifts T's high words in at the top.
#pragma once
#include "dmont.cuh"
#include "mont.cuh"

namespace xmpb {

// s = a^2 (2L words), one lane.
template <int L>
__device__ __forceinline__ void lane_square(uint32_t (&s)[2 * L], const uint32_t (&a)[L]) {
#pragma unroll
  for (int k = 0; k < 2 * L; k++) s[k] = 0;
#pragma unroll
  for (int i = 0; i < L - 1; i++) {
    uint64_t p[L];
#pragma unroll
    for (int j = i + 1; j < L; j++) p[j] = mul_wide(a[i], a[j]);
    // low halves at i + j, carry through s[i + L] into s[i + L + 1]
    s[2 * i + 1] = add_cc(s[2 * i + 1], (uint32_t)p[i + 1]);
#pragma unroll
    for (int j = i + 2; j < L; j++) s[i + j] = addc_cc(s[i + j], (uint32_t)p[j]);
    s[i + L] = addc_cc(s[i + L], 0u);
    s[i + L + 1] = addc(s[i + L + 1], 0u);
    // high halves at i + j + 1
    s[2 * i + 2] = add_cc(s[2 * i + 2], (uint32_t)(p[i + 1] >> 32));
#pragma unroll
    for (int j = i + 2; j < L; j++) s[i + j + 1] = addc_cc(s[i + j + 1], (uint32_t)(p[j] >> 32));
    s[i + L + 1] = addc(s[i + L + 1], 0u);
  }
  // double the cross products (their sum is below 2^(64L - 1)) and add the squares of the limbs
#pragma unroll
  for (int k = 2 * L - 1; k > 0; k--) s[k] = __funnelshift_l(s[k - 1], s[k], 1);
  s[0] <<= 1;
  uint64_t d[L];
#pragma unroll
  for (int i = 0; i < L; i++) d[i] = mul_wide(a[i], a[i]);
  s[0] = add_cc(s[0], (uint32_t)d[0]);
  s[1] = addc_cc(s[1], (uint32_t)(d[0] >> 32));
#pragma unroll
  for (int i = 1; i < L; i++) {
    s[2 * i] = addc_cc(s[2 * i], (uint32_t)d[i]);
    s[2 * i + 1] = addc_cc(s[2 * i + 1], (uint32_t)(d[i] >> 32));
  }
}

// One quotient row of the reduction: acc += N q (q from the lowest word), then the accumulator shifts down one
// word with `in` (a word of T) entering at the top.
template <int L>
__device__ __forceinline__ void redc_row(uint32_t (&r)[L], uint32_t &c0, uint32_t &c1, const uint32_t (&n)[L],
                                         uint32_t np0, uint32_t in) {
  const uint32_t q = r[0] * np0;
  uint64_t s[L];
  row_products<L>(s, n, q);
  add_low_halves<L>(r, c0, c1, s);
  add_high_halves<L>(r, c0, c1, s);
#pragma unroll
  for (int j = 0; j < L - 1; j++) r[j] = r[j + 1];
  r[L - 1] = add_cc(in, c0);
  c0 = addc_fma(c1);
  c1 = 0;
}

// Per-thread Montgomery squaring (TPI = 1).  r must not alias a.
template <int L>
__device__ __forceinline__ void mont_sqr1(const Group<1> &G, uint32_t (&r)[L], const uint32_t (&a)[L],
                                          const uint32_t (&n)[L], uint32_t np0) {
  uint32_t s[2 * L];
  lane_square<L>(s, a);
  uint32_t c0 = 0, c1 = 0;
#pragma unroll
  for (int k = 0; k < L; k++) r[k] = s[k];
#pragma unroll
  for (int i = 0; i < L; i++) redc_row<L>(r, c0, c1, n, np0, s[L + i]);
  // (r, c0) = (T + QN) / R < 2R: an overflow past R is removed by subtracting N
  dsub<1, L>(G, r, n, 0u - c0);
}

// ---- several lanes: the schedule of an even split -------------------------------------
//
// T lanes (T = 2, 4), lane g holding block A_g of L words.  Every lane computes, in one instruction stream,
// its own square S, the products P_r = 2 A_g A_{g+r mod T} for r = 1 .. T/2 - 1, and Q, the half of
// 2 A_g A_{g+T/2 mod T} that falls to it (lanes g < T/2 take their own low half against all of the partner's
// words, lanes g >= T/2 all of their own words against the partner's high half).  Block ids per lane: 0 S lo,
// 1 S hi, 2r and 2r + 1 the low and high blocks of P_r, T and T + 1 those of Q.  The functions say where each
// block belongs.  No kernel calls them (limbs: 4 x 8 was 5.7% faster than a general product and gave way to the
// digit kernels; digits: see powm_dig_sqr); the decomposition is kept with the test that proves it.

// T-word offset of block `id` of lane g (T lanes, L limbs each).
__host__ __device__ constexpr int sqr_block_offset(int T, int L, int g, int id) {
  if (id == 0) return 2 * g * L;
  if (id == 1) return 2 * g * L + L;
  if (id < T) {
    const int r = id / 2, h = (g + r) % T;
    return L * (g + h) + (id % 2 ? L : 0);
  }
  const int h = (g + T / 2) % T;
  return L * (g + h) + (g >= T / 2 ? L / 2 : 0) + (id == T ? 0 : L);
}

// The half-block boundary (row / (L/2)) at which lane g adds block `id` (independent of L).
__host__ __device__ constexpr int sqr_block_boundary(int T, int g, int id) {
  return (sqr_block_offset(T, 2, g, id) - 2 * g) / 1;
}

// This lane's schedule: nibble 2b + s = the id of its s-th block at boundary b (15: none).
struct SqrPlanBits {
  uint32_t w[3];  // 2 * (2T + 1) <= 18 nibbles for T <= 4
};

template <int T>
__host__ __device__ __forceinline__ SqrPlanBits sqr_lane_plan(uint32_t g) {
  static_assert(T == 2 || T == 4, "the lane plan holds 24 nibbles: two blocks at each of 2T + 1 boundaries");
  SqrPlanBits p;
  p.w[0] = p.w[1] = p.w[2] = 0xffffffffu;
  uint32_t used[2 * T + 1];
#pragma unroll
  for (int b = 0; b <= 2 * T; b++) used[b] = 0;
#pragma unroll
  for (int id = 0; id < T + 2; id++) {
    const uint32_t b = (uint32_t)sqr_block_boundary(T, (int)g, id);
    // slot = blocks already placed at this boundary (at most 2)
    uint32_t slot = 0;
#pragma unroll
    for (int bb = 0; bb <= 2 * T; bb++)
      if ((uint32_t)bb == b) slot = used[bb]++;
    const uint32_t nib = 2 * b + slot;
    const uint32_t word = nib / 8, sh = 4 * (nib % 8);
#pragma unroll
    for (int k = 0; k < 3; k++)
      if ((uint32_t)k == word) p.w[k] = (p.w[k] & ~(15u << sh)) | ((uint32_t)id << sh);
  }
  return p;
}

// Number of blocks the busiest lane adds at boundary b (the same in every lane), 2 bits per boundary.
__host__ __device__ constexpr uint64_t sqr_slots_mask(int T) {
  uint64_t mask = 0;
  for (int b = 0; b <= 2 * T; b++) {
    int most = 0;
    for (int g = 0; g < T; g++) {
      int c = 0;
      for (int id = 0; id < T + 2; id++)
        if (sqr_block_boundary(T, g, id) == b) c++;
      most = c > most ? c : most;
    }
    mask |= (uint64_t)most << (2 * b);
  }
  return mask;
}

// Limb kernels whose exponentiation squares with the specialised product: one lane, up to five limbs (more take
// the digit kernels, which have a square of their own).  They use the fixed window (every instance of a warp
// squares at the same steps; the sliding window is not combined with it).
__host__ __device__ constexpr bool powm_sqr(int TPI, int L) { return !powm_digits(TPI, L) && TPI == 1; }

// Dynamic shared memory of a 128-thread CTA of the register powm kernels: the digit kernels' operand B.
__host__ __device__ constexpr uint32_t powm_smem_bytes(int TPI, int L) { return 1024u * powm_digits(TPI, L); }

// r = a^2 R^-1 mod N (almost reduced) with the shape's squaring.  r must not alias a.
template <int TPI, int L>
__device__ __forceinline__ void mont_square(const Group<TPI> &G, uint32_t (&r)[L], const uint32_t (&a)[L],
                                            const uint32_t (&n)[L], uint32_t np0) {
  if constexpr (powm_sqr(TPI, L)) {
    mont_sqr1<L>(G, r, a, n, np0);
  } else {
    mont_mul<TPI, L>(G, r, a, a, n, np0);
  }
}

}  // namespace xmpb

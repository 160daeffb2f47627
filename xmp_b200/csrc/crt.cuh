// Fused CRT-RSA private operation, one kernel per batch (no counterpart in the
// reference library; it replaces the op sequence its CRT-RSA sample runs,
// samples/crt_rsa/rsa.cc:206-219: two mods, two powms, two muls, an add and a
// mod, each a separate launch with its own temporary arrays).
//
// Per instance, on a pair of groups of TPI lanes with L limbs each (n = TPI*L
// limbs = the precision of p and q, R = 2^(32n)), the first group working
// mod p and the second mod q:
//   1. Montgomery form of c mod p, for c of up to 2n limbs (c = c_hi R + c_lo):
//      Mont(c_lo, R^2) == c_lo R and Mont(c_hi, R^3) == c_hi R^2, each brought
//      below p, then added mod p.  The second group does the same mod q.
//   2. mp = c^dp mod p and, side by side, mq = c^dq mod q by fixed-window
//      exponentiation over max(precision of dp, dq) bits: the same number of
//      squarings and multiplies for every exponent (a zero window multiplies
//      by Mont(1)), so the schedule does not depend on the private exponent's
//      bits, and both groups of the pair run one instruction stream.
//   3. Garner's recombination on p: h = (mp - mq mod p) * qinv mod p, all in
//      Montgomery form, then m = mq + q*h as one 2n-limb product and sum.
// Nothing is stored between the steps except the window table (2^W entries
// in the scratch arena, as for powm); every intermediate stays in registers.
//
// Reducing a value y < R below an odd modulus N whose top bits may be clear
// uses Mont(Mont(y, R^2 mod N), 1), which is at most N, and one conditional
// subtraction (no division).
#pragma once
#include "powm_kernel.cuh"

namespace xmpb {

struct CrtArgs {
  ArrayView c, p, q, dp, dq, qinv;
  OutView out;
  uint32_t start;   // first op instance of this launch
  uint32_t count;   // op instances in this launch
  uint32_t window;  // fixed-window bits W
  uint32_t *table;  // per warp: crt_table_entries entries x 32 lanes x crt_slot_words words
};

// r += x over the group; returns the carry out of the top lane (same in every lane).
template <int TPI, int L>
__device__ __forceinline__ uint32_t dadd(const Group<TPI> &G, uint32_t (&r)[L], const uint32_t (&x)[L]) {
  r[0] = add_cc(r[0], x[0]);
#pragma unroll
  for (int k = 1; k < L; k++) r[k] = addc_cc(r[k], x[k]);
  uint32_t co = addc(0u, 0u);
  if (TPI == 1) return co;
  uint32_t ones = r[0];
#pragma unroll
  for (int k = 1; k < L; k++) ones &= r[k];
  uint32_t out;
  // a lane that carried out is not all ones (r + x <= 2^(32L+1) - 2), so generate and propagate are exclusive
  uint32_t ci = G.lookahead(co, ones == kFull, &out);
  r[0] = add_cc(r[0], ci);
#pragma unroll
  for (int k = 1; k < L; k++) r[k] = addc_cc(r[k], 0u);
  return out;
}

// r <- (r + x) mod N for r, x < N.
template <int TPI, int L>
__device__ __forceinline__ void dadd_mod(const Group<TPI> &G, uint32_t (&r)[L], const uint32_t (&x)[L],
                                         const uint32_t (&n)[L]) {
  uint32_t co = dadd<TPI, L>(G, r, x);
  uint32_t d[L];
#pragma unroll
  for (int k = 0; k < L; k++) d[k] = r[k];
  uint32_t bo = dsub<TPI, L>(G, d, n, kFull);
  bool take = co || !bo;
#pragma unroll
  for (int k = 0; k < L; k++) r[k] = take ? d[k] : r[k];
}

// r <- (r - x) mod N for r, x < N.
template <int TPI, int L>
__device__ __forceinline__ void dsub_mod(const Group<TPI> &G, uint32_t (&r)[L], const uint32_t (&x)[L],
                                         const uint32_t (&n)[L]) {
  uint32_t bo = dsub<TPI, L>(G, r, x, kFull);
  uint32_t z[L];
#pragma unroll
  for (int k = 0; k < L; k++) z[k] = 0;
  // add N back when the difference went negative (the carry out cancels the borrow)
  uint32_t nm[L];
#pragma unroll
  for (int k = 0; k < L; k++) nm[k] = bo ? n[k] : z[k];
  dadd<TPI, L>(G, r, nm);
}

// y <- y mod N for any y < R: Mont(y, R^2) == y R, Mont(that, 1) <= N, then one conditional subtraction.
template <int TPI, int L>
__device__ __forceinline__ void dcanon(const Group<TPI> &G, uint32_t (&y)[L], const uint32_t (&n)[L], uint32_t np0,
                                       const uint32_t (&r2)[L]) {
  uint32_t t[L], one[L];
  mont_mul<TPI, L>(G, t, y, r2, n, np0);
#pragma unroll
  for (int k = 0; k < L; k++) one[k] = (G.lane == 0 && k == 0) ? 1u : 0u;
  mont_mul<TPI, L>(G, y, t, one, n, np0);
  dreduce<TPI, L>(G, y, n);
}

// Montgomery form (canonical, below N) of c mod N for c = c_hi R + c_lo.
template <int TPI, int L>
__device__ __forceinline__ void crt_reduce(const Group<TPI> &G, uint32_t (&xm)[L], const uint32_t (&clo)[L],
                                           const uint32_t (&chi)[L], const uint32_t (&n)[L], uint32_t np0,
                                           const uint32_t (&r2)[L]) {
  uint32_t r3[L], u[L];
  mont_mul<TPI, L>(G, r3, r2, r2, n, np0);  // R^3 mod N (below R)
  mont_mul<TPI, L>(G, u, chi, r3, n, np0);  // == c_hi R^2
  dcanon<TPI, L>(G, u, n, np0, r2);
  mont_mul<TPI, L>(G, xm, clo, r2, n, np0);  // == c_lo R
  dcanon<TPI, L>(G, xm, n, np0, r2);
  dadd_mod<TPI, L>(G, xm, u, n);
}

// acc <- Mont(x^e) for the exponent element `ee` scanned over its whole precision in W-bit windows;
// xm = Mont(x) below N.  Table slot e holds Mont(x^e), e < 2^W (slot 0 = R - N, Mont(1)).
template <int TPI, int L>
__device__ __forceinline__ void powm_fixed_full(const Group<TPI> &G, uint32_t (&acc)[L], const uint32_t (&xm)[L],
                                                const ArrayView &ex, uint32_t ee, uint32_t nbits,
                                                const uint32_t (&n)[L], uint32_t np0, uint32_t W, uint32_t *slot) {
  const size_t es = (size_t)32 * L;
  uint32_t t[L], y[L];
#pragma unroll
  for (int k = 0; k < L; k++) t[k] = 0;
  dsub<TPI, L>(G, t, n, kFull);
  slot_store<L>(slot, t);
  slot_store<L>(slot + es, xm);
#pragma unroll
  for (int k = 0; k < L; k++) acc[k] = xm[k];
  const uint32_t entries = 1u << W;
#pragma unroll 1
  for (uint32_t e = 2; e < entries; e++) {
    mont_mul<TPI, L>(G, t, acc, xm, n, np0);
#pragma unroll
    for (int k = 0; k < L; k++) acc[k] = t[k];
    slot_store<L>(slot + e * es, acc);
  }
  const uint32_t nwin = (nbits + W - 1) / W;  // bits past the exponent's precision read as zero
  uint32_t win = exp_window(ex, ee, (nwin - 1) * W, W);
  slot_load<L>(slot + win * es, acc);
#pragma unroll 1
  for (int32_t wi = (int32_t)nwin - 2; wi >= 0; wi--) {
    win = exp_window(ex, ee, (uint32_t)wi * W, W);
#pragma unroll 1
    for (uint32_t s = 0; s < W; s++) {
      mont_square<TPI, L>(G, t, acc, n, np0);
#pragma unroll
      for (int k = 0; k < L; k++) acc[k] = t[k];
    }
    slot_load<L>(slot + win * es, y);
    mont_mul<TPI, L>(G, t, acc, y, n, np0);
#pragma unroll
    for (int k = 0; k < L; k++) acc[k] = t[k];
  }
}

// (lo, hi) <- a * b over the group: the 2n-limb product, lane g holding limbs
// [gL, gL + L) of the low half and of the high half.  Rows of a * b_i on a
// shifting accumulator (as in mont_mul, without the reduction): after row i
// the group's lowest word is final product word i and goes to its owner lane.
template <int TPI, int L>
__device__ __forceinline__ void dmul_wide(const Group<TPI> &G, uint32_t (&lo)[L], uint32_t (&hi)[L],
                                          const uint32_t (&a)[L], const uint32_t (&b)[L]) {
  uint32_t r[L], c0 = 0, c1 = 0;
#pragma unroll
  for (int k = 0; k < L; k++) {
    r[k] = 0;
    lo[k] = 0;
  }
#pragma unroll 1
  for (int src = 0; src < TPI; src++) {
#pragma unroll
    for (int k = 0; k < L; k++) {
      const uint32_t w = G.bcast(b[k], src);
      uint64_t p[L];
      row_products<L>(p, a, w);
      add_low_halves<L>(r, c0, c1, p);
      add_high_halves<L>(r, c0, c1, p);
      const uint32_t fin = G.bcast(r[0], 0);
      if (G.lane == (uint32_t)src) lo[k] = fin;
      const uint32_t t = G.from_next(r[0]);
#pragma unroll
      for (int j = 0; j < L - 1; j++) r[j] = r[j + 1];
      r[L - 1] = add_cc(t, c0);
      c0 = addc_fma(c1);
      c1 = 0;
    }
  }
  dnormalize<TPI, L>(G, r, c0);  // carry out of the top lane is zero: a * b < R^2
#pragma unroll
  for (int k = 0; k < L; k++) hi[k] = r[k];
}

// Limbs [off + lane*L, off + lane*L + L) of element e.
template <int TPI, int L>
__device__ __forceinline__ void load_lane_limbs_at(uint32_t (&x)[L], const ArrayView &v, uint32_t e, uint32_t lane,
                                                   uint32_t off) {
  const uint32_t j0 = off + lane * L;
  if (L % 4 == 0 && off % 4 == 0) {
#pragma unroll
    for (int m = 0; m < L / 4; m++) {
      uint4 g = load_group(v.limbs, v.nlimbs, v.stride, e, j0 / 4 + m);
      x[4 * m] = g.x;
      x[4 * m + 1] = g.y;
      x[4 * m + 2] = g.z;
      x[4 * m + 3] = g.w;
    }
  } else {
#pragma unroll
    for (int k = 0; k < L; k++) x[k] = load_limb(v.limbs, v.nlimbs, v.stride, e, j0 + k);
  }
}

template <int TPI, int L>
__device__ __forceinline__ void store_lane_limbs_at(const uint32_t (&x)[L], const OutView &v, uint32_t e,
                                                    uint32_t lane, uint32_t off) {
  const uint32_t j0 = off + lane * L;
  if (L % 4 == 0 && off % 4 == 0) {
#pragma unroll
    for (int m = 0; m < L / 4; m++) {
      uint32_t g = j0 / 4 + m;
      if (g * 4 < v.nlimbs)
        store_group(v.limbs, v.nlimbs, v.stride, e, g, make_uint4(x[4 * m], x[4 * m + 1], x[4 * m + 2], x[4 * m + 3]));
    }
  } else {
#pragma unroll
    for (int k = 0; k < L; k++)
      if (j0 + k < v.nlimbs) limb_ref(v.limbs, v.stride, e, j0 + k) = x[k];
  }
}

// Modulus constants of element e of `mv`: N, n0' and R^2 mod N.
template <int TPI, int L>
__device__ __forceinline__ uint32_t crt_modulus(const Group<TPI> &G, uint32_t (&n)[L], uint32_t (&r2)[L],
                                                const ArrayView &mv, uint32_t e) {
  load_lane_limbs_at<TPI, L>(n, mv, e, G.lane, 0);
  const uint32_t np0 = neg_inv32(G.bcast(n[0], 0));
  compute_r2<TPI, L>(G, r2, n, np0);
  return np0;
}

// ---- the same on 52-bit digits (dmont.cuh) -------------------------------------------

// r = the balanced digits of the signed 64-bit digits d (|d| < 2^63, value within +-R / 4).
template <int TPI, int D>
__device__ __forceinline__ void dig_balance(const Group<TPI> &G, double (&r)[D], const int64_t (&d)[D]) {
  uint64_t col[D];
#pragma unroll
  for (int j = 0; j < D; j++) col[j] = (uint64_t)d[j];
  dig_settle<TPI, D>(G, r, col, 0u, 0u);
}

// The group's 2N canonical digits of add + a * B (B in shared memory, a balanced; add, and the sum, not
// negative) into out[0 .. 2N).  Rows as in dig_mul without the reduction: column 0 of row i is product
// digit i once its constant is taken off, and carries into the next column.
template <int TPI, int D>
__device__ __forceinline__ void dig_mul_add_wide(const Group<TPI> &G, uint64_t *out, const int64_t (&add)[D],
                                                 const double (&a)[D], const DigSmem &sm) {
  constexpr int N = TPI * D;
  constexpr uint64_t kLo = (uint64_t)kDigLoBits << 52, kHi = (0x467ull << 52) + (1ull << 51);
  const double *bp = dig_b<TPI, D>(sm);
  uint64_t col[D + 1], k = kLo;
#pragma unroll
  for (int j = 0; j < D; j++) col[j] = (uint64_t)add[j];
  col[D] = 0;
#pragma unroll 1
  for (int i = 0; i < N; i++) {
    dig_row<D, 0>(col, a, bp[i * (32 / TPI)]);
    const int64_t v = (int64_t)(col[0] - k);
    k += kLo + kHi;
    if (G.lane == 0) out[i] = (uint64_t)v & kDigMask;
    uint64_t next = 0;
    if (TPI > 1) {
      next = __shfl_down_sync(kFull, col[0], 1, TPI);
      if (G.lane == TPI - 1) next = 0;
    }
#pragma unroll
    for (int j = 0; j < D; j++) col[j] = col[j + 1];
    col[D] = 0;
    col[D - 1] += next;
    if (G.lane == 0) col[0] += (uint64_t)(v >> 52);
  }
  int64_t d[D];
#pragma unroll
  for (int j = 0; j < D; j++) {
    const uint64_t p = G.lane * D + j;
    d[j] = (int64_t)(col[j] - (N - 1 - p) * kLo - (N - p) * kHi);
  }
  dig_carry<TPI, D>(G, d);
#pragma unroll
  for (int j = 0; j < D; j++) out[N + G.lane * D + j] = (uint64_t)d[j];
  __syncwarp();
}

// Steps 1-3 above.  Differences from the limb form: c splits at R = 2^(52N) (its low part balanced, so
// within R / 2), the two parts' Montgomery forms are added without reducing (below 2N, R >= 16N), and
// Garner's difference mp - mq goes into the product by qinv signed and unreduced (R >= 16 max(p, q)).
// R^2 waits in the table's last entry.
template <int TPI, int L, int D>
__device__ __forceinline__ void dig_crt_instance(const Group<TPI> &G, const CrtArgs &a, uint32_t i, bool valid,
                                                 bool second, double *tab, const DigSmem &sm) {
  static_assert(52 * TPI * D >= 32 * TPI * L + 4, "R >= 16 N");
  constexpr int N = TPI * D;
  const ArrayView mv = second ? a.q : a.p, ov = second ? a.p : a.q, ev = second ? a.dq : a.dp;
  const uint32_t em = in_element(mv, i), W = a.window;
  const uint32_t nwin = (max(a.dp.nlimbs, a.dq.nlimbs) * 32 + W - 1) / W;
  double n[D], t[D], acc[D];
  uint64_t np;
  dig_load<TPI, D>(G, n, mv.limbs, mv.nlimbs, mv.stride, em);
  {
    uint32_t nl[L];
    load_lane_limbs_at<TPI, L>(nl, mv, em, G.lane, 0);
    np = dig_neg_inv(nl[0], nl[1]);
    dig_r2<TPI, L, D>(G, t, nl, n, np, sm);
  }
  dig_slot_store<TPI, D>(tab, 1u << W, t);
  dig_set_b<TPI, D>(G, sm, t);
  {
    double one[D];
#pragma unroll
    for (int k = 0; k < D; k++) one[k] = (G.lane == 0 && k == 0) ? 1.0 : 0.0;
    dig_mul<TPI, D>(G, one, one, sm, n, np);
    dig_slot_store<TPI, D>(tab, 0, one);  // Mont(1)
  }
  {
    const uint32_t ec = in_element(a.c, i);
    double u[D];
    dig_mul<TPI, D>(G, t, t, sm, n, np);  // R^3
    dig_load<TPI, D>(G, acc, a.c.limbs, a.c.nlimbs, a.c.stride, ec);
    dig_mul<TPI, D>(G, acc, acc, sm, n, np);  // c_lo R
    dig_set_b<TPI, D>(G, sm, t);
    dig_load<TPI, D>(G, u, a.c.limbs, a.c.nlimbs, a.c.stride, ec, N);
    dig_mul<TPI, D>(G, u, u, sm, n, np);  // c_hi R^2
    int64_t d[D];
#pragma unroll
    for (int k = 0; k < D; k++) d[k] = (int64_t)acc[k] + (int64_t)u[k];
    dig_balance<TPI, D>(G, t, d);
  }
  dig_slot_store<TPI, D>(tab, 1, t);
  const uint32_t ee = in_element(ev, i);
  dig_fixed_table<TPI, D>(G, acc, t, n, np, W, tab, sm);
  dig_fixed_scan<TPI, L, D, false>(G, acc, ev, ee, nwin, W, n, np, tab, sm);
#pragma unroll
  for (int k = 0; k < D; k++) t[k] = (G.lane == 0 && k == 0) ? 1.0 : 0.0;
  dig_set_b<TPI, D>(G, sm, t);
  dig_mul<TPI, D>(G, acc, acc, sm, n, np);
  int64_t mine[D], other[D];
  dig_canon<TPI, D>(G, mine, acc, n);
#pragma unroll
  for (int k = 0; k < D; k++) other[k] = (int64_t)__shfl_xor_sync(kFull, (unsigned long long)mine[k], TPI);
  dig_slot_load<TPI, D>(tab, 1u << W, t);
  dig_set_b<TPI, D>(G, sm, t);
  dig_load<TPI, D>(G, t, a.qinv.limbs, a.qinv.nlimbs, a.qinv.stride, in_element(a.qinv, i));
  dig_mul<TPI, D>(G, t, t, sm, n, np);  // qinv R
  dig_set_b<TPI, D>(G, sm, t);
#pragma unroll
  for (int k = 0; k < D; k++) mine[k] -= other[k];
  dig_balance<TPI, D>(G, acc, mine);
  dig_mul<TPI, D>(G, acc, acc, sm, n, np);  // (mp - mq) qinv mod p
  dig_canon<TPI, D>(G, mine, acc, n);       // h
  dig_balance<TPI, D>(G, t, mine);
  dig_set_b<TPI, D>(G, sm, t);
  dig_load<TPI, D>(G, t, ov.limbs, ov.nlimbs, ov.stride, in_element(ov, i));
  // the table is done with: its first 2N digits per group take m = mq + q h
  uint64_t *st = reinterpret_cast<uint64_t *>(tab) + (size_t)((threadIdx.x & 31) / TPI) * (2 * N);
  __syncwarp();
  dig_mul_add_wide<TPI, D>(G, st, other, t, sm);
  if (valid && !second) {
    const uint32_t o = out_element(a.out, i);
    if (o < a.out.count)
      for (uint32_t g = G.lane; g < div_up(a.out.nlimbs, 4); g += TPI)
        store_group(a.out.limbs, a.out.nlimbs, a.out.stride, o, g, dig_group(st, 2 * N, g));
  }
}

// Words per lane and entries of the window table (the digit form keeps R^2 in one more).
__host__ __device__ constexpr uint32_t crt_slot_words(int L, int D) { return D ? 2 * D : L; }
__host__ __device__ constexpr uint32_t crt_table_entries(int D, uint32_t W) { return (1u << W) + (D ? 1u : 0u); }

// The two exponentiations of an instance run side by side on two adjacent
// groups of one warp (lanes [0, TPI) of the pair work mod p, lanes
// [TPI, 2 TPI) mod q), so a batch has twice as many independent groups as
// instances and each group does one exponentiation: measured on limbs at
// 16,384 RSA-2048 operations (4 lanes x 8 limbs), 17.8 ms against 21.6 ms
// with both exponentiations on one group in turn, and at 1,024 operations
// (8 x 4) 2.0 ms against 4.1 ms.  The results meet with one shuffle per limb
// (lane l and l ^ TPI hold the same limbs of mp and mq); both groups then run
// the same Garner steps on their own modulus -- the first group's are
// h = (mp - mq mod p) * qinv mod p and m = mq + q h, which it stores; the
// second group's mirror image is discarded.
// D: the powm kernels' digits, or 0 for limbs, with their bound on CTAs per SM, at which this kernel's longer
// state spills up to 208 bytes a thread.  With one CTA fewer (two at least) RSA-4096 x 2,048 takes 11.3 ms
// instead of 12.3, RSA-2048 x 4,096 3.13 instead of 3.37, x 16,384 10.9 instead of 10.8: the bound was not fitted here.
template <int TPI, int L, int D>
__global__ void __launch_bounds__(128, D ? powm_min_blocks(TPI, L) : 1) crt_kernel(CrtArgs a) {
  static_assert(TPI <= 16, "both groups of a pair sit in one warp");
  const DigSmem sm = powm_smem_setup<TPI, L>();
  Group<TPI> G;
  const uint32_t gtid = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t local = gtid / (2 * TPI);
  const bool second = ((gtid / TPI) & 1u) != 0;  // this group works mod q
  const bool valid = local < a.count;
  // pairs past the end run a copy of the last instance so every shuffle sees a full warp
  const uint32_t i = a.start + (valid ? local : a.count - 1);
  uint32_t *table = a.table + (size_t)(gtid >> 5) * ((size_t)32 * crt_slot_words(L, D) * crt_table_entries(D, a.window));
  if constexpr (D > 0) {
    dig_crt_instance<TPI, L, D>(G, a, i, valid, second, reinterpret_cast<double *>(table), sm);
    return;
  } else {
  uint32_t *const slot = table + (size_t)(threadIdx.x & 31) * L;
  const ArrayView mv = second ? a.q : a.p, ov = second ? a.p : a.q, ev = second ? a.dq : a.dp;
  const uint32_t em = in_element(mv, i);
  const uint32_t nbits = max(a.dp.nlimbs, a.dq.nlimbs) * 32;
  const uint32_t n_limbs = TPI * L;

  uint32_t n[L], r2[L], xm[L];
  uint32_t np0;
  {
    uint32_t clo[L], chi[L];
    const uint32_t ec = in_element(a.c, i);
    load_lane_limbs_at<TPI, L>(clo, a.c, ec, G.lane, 0);
    load_lane_limbs_at<TPI, L>(chi, a.c, ec, G.lane, n_limbs);
    np0 = crt_modulus<TPI, L>(G, n, r2, mv, em);
    crt_reduce<TPI, L>(G, xm, clo, chi, n, np0, r2);
  }
  uint32_t one[L], acc[L], mine[L], other[L];
#pragma unroll
  for (int k = 0; k < L; k++) one[k] = (G.lane == 0 && k == 0) ? 1u : 0u;
  powm_fixed_full<TPI, L>(G, acc, xm, ev, in_element(ev, i), nbits, n, np0, a.window, slot);
  mont_mul<TPI, L>(G, mine, acc, one, n, np0);
  dreduce<TPI, L>(G, mine, n);
#pragma unroll
  for (int k = 0; k < L; k++) other[k] = __shfl_xor_sync(kFull, mine[k], TPI);
  // Garner on this group's modulus (p for the first group)
  uint32_t h[L];
  {
    compute_r2<TPI, L>(G, r2, n, np0);
    uint32_t d[L], t[L], u[L];
#pragma unroll
    for (int k = 0; k < L; k++) d[k] = other[k];
    dcanon<TPI, L>(G, d, n, np0, r2);  // mq mod p
#pragma unroll
    for (int k = 0; k < L; k++) t[k] = mine[k];
    dsub_mod<TPI, L>(G, t, d, n);  // D = (mp - mq) mod p
    mont_mul<TPI, L>(G, d, t, r2, n, np0);  // == D R
    load_lane_limbs_at<TPI, L>(u, a.qinv, in_element(a.qinv, i), G.lane, 0);
    mont_mul<TPI, L>(G, t, u, r2, n, np0);  // == qinv R
    mont_mul<TPI, L>(G, u, d, t, n, np0);   // == D qinv R
    mont_mul<TPI, L>(G, h, u, one, n, np0);  // == D qinv, at most p
    dreduce<TPI, L>(G, h, n);
  }
  // m = mq + q h (below pq)
  uint32_t lo[L], hi[L];
  load_lane_limbs_at<TPI, L>(n, ov, in_element(ov, i), G.lane, 0);
  dmul_wide<TPI, L>(G, lo, hi, n, h);
  uint32_t co = dadd<TPI, L>(G, lo, other);
  uint32_t cw[L];
#pragma unroll
  for (int k = 0; k < L; k++) cw[k] = (G.lane == 0 && k == 0) ? co : 0u;
  dadd<TPI, L>(G, hi, cw);
  if (valid && !second) {
    const uint32_t o = out_element(a.out, i);
    if (o < a.out.count) {
      store_lane_limbs_at<TPI, L>(lo, a.out, o, G.lane, 0);
      store_lane_limbs_at<TPI, L>(hi, a.out, o, G.lane, n_limbs);
    }
  }
  }
}

}  // namespace xmpb

// Host side of the fused CRT-RSA operation (crt.cuh): kernel registry, the
// configuration rule, and xmpIntegersPowmCRT[Async] (declared in
// include/xmp_b200.h; no counterpart in the reference library).
#include "crt.h"
#include "../../include/xmp_b200.h"
#include <algorithm>
#include <vector>

namespace xmpb {

std::vector<CrtKernelEntry> &crt_registry() {
  static std::vector<CrtKernelEntry> r;
  return r;
}

#define XMPB_REGISTER_CRT_AS(TPI, L, D, NAME)                                                    \
  static void crt_launch_##NAME(const CrtArgs &a, int grid, int threads, cudaStream_t s) {       \
    crt_kernel<TPI, L, D><<<grid, threads, powm_smem_bytes(TPI, L), s>>>(a);                      \
  }                                                                                               \
  static CrtKernelRegistrar crt_reg_##NAME(TPI, L, D, crt_launch_##NAME);
#define XMPB_REGISTER_CRT(TPI, L) XMPB_REGISTER_CRT_AS(TPI, L, powm_digits(TPI, L), TPI##_##L)

// Shapes for halves of 256 to 4096 bits (RSA-512 to RSA-8192): two or more per size, from the fewest lanes
// (digit kernels: most throughput) to the shortest latency.
XMPB_REGISTER_CRT(4, 2)
XMPB_REGISTER_CRT(8, 1)
XMPB_REGISTER_CRT(1, 16)
XMPB_REGISTER_CRT(4, 4)
XMPB_REGISTER_CRT(8, 2)
XMPB_REGISTER_CRT(1, 24)
XMPB_REGISTER_CRT(4, 6)
XMPB_REGISTER_CRT(8, 3)
XMPB_REGISTER_CRT(1, 32)
XMPB_REGISTER_CRT(2, 16)
XMPB_REGISTER_CRT(4, 8)
XMPB_REGISTER_CRT(8, 4)
XMPB_REGISTER_CRT(2, 24)
XMPB_REGISTER_CRT(4, 12)
XMPB_REGISTER_CRT(8, 6)
// limbs too: a lone row of six is 10% shorter than four digits' (3072-bit keys, 593 to 1,184 at once, 5.05 / 5.72 ms)
XMPB_REGISTER_CRT_AS(8, 6, 0, 8_6_limbs)
XMPB_REGISTER_CRT(16, 3)
XMPB_REGISTER_CRT(4, 16)
XMPB_REGISTER_CRT(8, 8)
XMPB_REGISTER_CRT(16, 4)
XMPB_REGISTER_CRT(4, 24)
XMPB_REGISTER_CRT(8, 12)
XMPB_REGISTER_CRT(16, 6)
XMPB_REGISTER_CRT(8, 16)
XMPB_REGISTER_CRT(16, 8)

// The shape with the lowest expected time for the batch (two lane groups an instance).
CrtConfig crt_config(uint32_t nlimbs, uint32_t exp_bits, uint32_t count, uint32_t sm_count) {
  CrtConfig best;
  double best_score = 1e300;
  for (const auto &e : crt_registry()) {
    if ((uint32_t)(e.tpi * e.limbs) < nlimbs) continue;
    const double score = powm_shape_cycles(e.tpi, e.limbs, 2.0 * count, sm_count, e.digits);
    if (score < best_score) {
      best_score = score;
      best.tpi = e.tpi;
      best.limbs = e.limbs;
      best.digits = e.digits;
      best.launch = e.launch;
    }
  }
  best.window = window_for_bits(exp_bits, false);
  return best;
}

size_t crt_table_bytes(const CrtConfig &c, uint32_t count) {
  const size_t threads =
      round_up((uint32_t)std::min<uint64_t>((uint64_t)count * c.tpi * 2, 0xffffff80ull), (uint32_t)c.threads);
  return threads * (size_t)crt_slot_words(c.limbs, c.digits) * crt_table_entries(c.digits, (uint32_t)c.window) * 4;
}

uint32_t crt_chunk_for(const CrtConfig &c, size_t limit, uint32_t count) {
  const uint32_t per_block = c.threads / (2 * c.tpi);  // a pair of groups per instance
  const size_t per_inst = (size_t)2 * c.tpi * crt_slot_words(c.limbs, c.digits) * crt_table_entries(c.digits, (uint32_t)c.window) * 4;
  const uint64_t fit = std::min<uint64_t>(limit / per_inst, (1ull << 31) / (2 * c.tpi)) / per_block * per_block;
  return fit < per_block ? 0u : (uint32_t)std::min<uint64_t>(count, fit);
}

// Bytes of one warp's window-1 table, the least a shape can run with.
static size_t crt_least_bytes(int limbs, int digits) {
  return (size_t)32 * crt_slot_words(limbs, digits) * crt_table_entries(digits, 1) * 4;
}

uint32_t crt_fit(CrtConfig &c, uint32_t nlimbs, size_t limit, uint32_t count) {
  uint32_t chunk;
  while ((chunk = crt_chunk_for(c, limit, count)) == 0) {
    if (c.window > 1) {
      c.window--;
    } else if (c.threads > 32) {
      c.threads = 32;
    } else {
      // The shape was chosen for its speed (one lane of 20 digits takes 15 KB); the limit decides before that.
      const size_t least = crt_least_bytes(c.limbs, c.digits);
      size_t best = least;
      for (const auto &e : crt_registry()) {
        if ((uint32_t)(e.tpi * e.limbs) < nlimbs || crt_least_bytes(e.limbs, e.digits) >= best) continue;
        best = crt_least_bytes(e.limbs, e.digits);
        c.tpi = e.tpi;
        c.limbs = e.limbs;
        c.digits = e.digits;
        c.launch = e.launch;
      }
      if (best == least) return 0;
    }
  }
  return chunk;
}

void crt_launch(const CrtConfig &c, CrtArgs a, uint32_t count, uint32_t chunk, cudaStream_t s) {
  for (uint32_t start = 0; start < count; start += chunk) {
    a.start = start;
    a.count = std::min(chunk, count - start);
    c.launch(a, grid_for((uint64_t)a.count * c.tpi * 2, c.threads), c.threads, s);
  }
}

xmpError_t crt_validate(xmpHandle_t h, xmpIntegers_t out, xmpIntegers_t c, xmpIntegers_t p, xmpIntegers_t q,
                        xmpIntegers_t dp, xmpIntegers_t dq, xmpIntegers_t qinv, uint32_t count) {
  if (!h || !out || !c || !p || !q || !dp || !dq || !qinv) return xmpErrorInvalidParameter;
  for (xmpIntegers_t x : {out, c, p, q, dp, dq, qinv})
    if (x->device != h->device) return xmpErrorInvalidDevice;
  if (out->count < count) return xmpErrorInvalidCount;
  const uint32_t hb = p->precision;
  if (q->precision != hb || qinv->precision != hb || out->precision != 2 * hb || c->precision > 2 * hb)
    return xmpErrorInvalidPrecision;
  return xmpErrorSuccess;
}

CrtArgs crt_args(xmpIntegers_t out, uint32_t *out_limbs, xmpIntegers_t c, xmpIntegers_t p, xmpIntegers_t q,
                 xmpIntegers_t dp, xmpIntegers_t dq, xmpIntegers_t qinv) {
  CrtArgs a;
  a.c = view_in(c);
  a.p = view_in(p);
  a.q = view_in(q);
  a.dp = view_in(dp);
  a.dq = view_in(dq);
  a.qinv = view_in(qinv);
  a.out = view_out(out, out_limbs, nullptr);
  a.start = 0;
  a.count = 0;
  a.window = 0;
  a.table = nullptr;
  return a;
}

}  // namespace xmpb

using namespace xmpb;

extern "C" {

xmpError_t XMPAPI xmpIntegersPowmCRTAsync(xmpHandle_t h, xmpIntegers_t out, const xmpIntegers_t c,
                                          const xmpIntegers_t p, const xmpIntegers_t q, const xmpIntegers_t dp,
                                          const xmpIntegers_t dq, const xmpIntegers_t qinv, uint32_t count) {
  xmpError_t e = crt_validate(h, out, c, p, q, dp, dq, qinv, count);
  if (e != xmpErrorSuccess) return e;
  if (count == 0) return xmpErrorSuccess;
  DeviceGuard guard(h->device);
  CrtConfig cfg = crt_config(p->nlimbs, std::max(dp->precision, dq->precision), count, h->sm_count);
  if (!cfg.launch) return xmpErrorUnsupported;
  // chunk so the window tables fit the scratch limit; shrink the window when one block does not fit
  const uint32_t chunk = crt_fit(cfg, p->nlimbs, scratch_limit(h), count);
  if (chunk == 0) return xmpErrorIncreaseScratchLimit;
  // an output that is also an input is written through the handle's temporary output buffer
  const bool aliased = (out == c || out == p || out == q || out == dp || out == dq || out == qinv);
  OutTarget t;
  if ((e = begin_output(h, out, aliased, aliased, &t)) != xmpErrorSuccess) return e;
  if ((e = ensure_scratch(h, crt_table_bytes(cfg, chunk))) != xmpErrorSuccess) return e;
  CrtArgs a = crt_args(out, t.limbs, c, p, q, dp, dq, qinv);
  a.window = (uint32_t)cfg.window;
  a.table = (uint32_t *)h->scratch;
  crt_launch(cfg, a, count, chunk, h->stream);
  if ((e = check_cuda()) != xmpErrorSuccess) return e;
  return end_output(h, out, t);
}

xmpError_t XMPAPI xmpIntegersPowmCRT(xmpHandle_t h, xmpIntegers_t out, const xmpIntegers_t c, const xmpIntegers_t p,
                                     const xmpIntegers_t q, const xmpIntegers_t dp, const xmpIntegers_t dq,
                                     const xmpIntegers_t qinv, uint32_t count) {
  xmpError_t e = xmpIntegersPowmCRTAsync(h, out, c, p, q, dp, dq, qinv, count);
  if (e != xmpErrorSuccess) return e;
  DeviceGuard guard(h->device);
  if (cudaStreamSynchronize(h->stream) != cudaSuccess) return xmpErrorCuda;
  return check_cuda();
}

}  // extern "C"

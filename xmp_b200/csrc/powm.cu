// Host dispatch of xmpIntegersPowm[Async] (replaces src/powm.cu:61-307 and
// src/include/powm_operators.h:15-455).  Validation and index semantics are the
// reference's: out/base/mod precisions equal, exponent precision free, output
// index = indices[0][i], base/exp/mod = indices[1..3][i % n] % array count.
// The configuration (distribution, lanes per instance, limbs per lane, window)
// comes from the handle's tuner when it has an entry for the size class,
// otherwise from a register/occupancy heuristic; the reference's static
// Maxwell/Kepler latency tables (powm.cu:120-236) have no counterpart.
#include "powm.h"
#include "../../include/xmp_b200.h"
#include <algorithm>
#include <math.h>

using namespace xmpb;

namespace xmpb {

std::vector<PowmKernelEntry> &powm_registry() {
  static std::vector<PowmKernelEntry> r;
  return r;
}

const PowmKernelEntry *powm_find(int tpi, int limbs) {
  for (const auto &e : powm_registry())
    if (e.tpi == tpi && e.limbs == limbs) return &e;
  return nullptr;
}

int window_for_bits(uint32_t exp_bits, bool sliding) {
  if (exp_bits <= 1) return 1;
  int best = 1;
  double best_cost = 1e300;
  for (int w = 1; w <= 7; w++) {
    // sliding: the table build is weighted 5/4 (its entries are also stored; on B200 this puts the
    // 2048-bit choice on W = 6, measured 0.45% faster than W = 7, and keeps 1024 -> 6, 4096 -> 7)
    double cost = sliding ? 1.25 * (double)(1 << (w - 1)) + ceil((double)exp_bits / (w + 1))
                          : (double)((1 << w) - 2) + ceil((double)exp_bits / w);
    if (cost < best_cost - 1e-9) {
      best_cost = cost;
      best = w;
    }
  }
  return best;
}

bool powm_cta_preferred(uint32_t nlimbs, uint32_t count, uint32_t sm_count) {
  const uint32_t limbs = powm_cta_limbs(nlimbs);
  // Up to 512 bits the smallest CTA (1024-bit operands) pads too much: it ties with the lane kernels at 512
  // bits (0.55 ms for 148 instances, 0.59 ms for 296, vs 0.59 ms on 4 x 4) and loses below (148 instances of 384
  // bits 0.43 ms vs 0.33 on 4 x 3, 256 bits 0.32 vs 0.15 on 1 x 8).  From 544 bits on it is faster alone at every measured size (544: 0.57 vs 1.11 ms on 8 x 4,
  // 1056: 1.40 vs 2.86, 1536: 1.97 vs 4.04, 2048: 2.56 vs 7.6, 3072: 5.94 vs 15.6, 4096: 9.7 vs 29.3 ms).
  if (!limbs || nlimbs <= 16) return false;
  // A CTA per instance runs it near its lone latency while the SMs hold the batch; the lane kernels
  // need thousands of instances before their throughput beats that.  Measured on B200 (full-length
  // exponents), CTA at 148 / 296 / 444 / 592 / 888 instances vs the best lane kernel: 768 bits
  // 0.78/0.84/0.91/0.97/1.20 vs 1.11 ms; 1024 bits 0.99/1.07/1.17/1.25/1.54 vs 2.03 ms; 1536 bits
  // 1.98/2.51/4.35 vs 4.03 ms; 2048 bits 2.58/3.27/5.68/6.52 vs 7.7 ms; 3072 bits 5.98/11.9 vs 15.6 ms;
  // 4096 bits 9.8/19.5 vs 29.5 ms.  The limits are older than these times and not fitted to them: above 2048 bits
  // two CTAs per SM and at 2048 bits four would gain as well.
  uint32_t per_sm = 1;
  if (limbs == 32) per_sm = nlimbs > 24 ? 6 : 4;
  else if (limbs == 64) per_sm = nlimbs > 48 ? 3 : 2;
  return count <= per_sm * sm_count;
}

// A product is TPI * L limb rows or TPI * D digit rows.  Fitted to every registered shape's time on B200
// (512-bit exponents; one instance, and 151,552 / TPI): a digit row of D digits takes max(155 + 8 D, 21.5 D)
// cycles alone and 38 + 17.5 D of a full scheduler (measured / fitted: D = 5 133 / 126, 8 178 / 178, 10 212 / 213, 15
// 293 / 301, 20 396 / 388; alone D = 4 184 / 187, 5 195 / 195, 8 215 / 219, 10 237 / 235, 15 314 / 322, 20 434 / 430); a limb
// row max(100, 80 + 5 L) and 10 + 13.5 L (L = 6 92 / 91, 4 68 / 64, 2 42 / 37; alone L = 6 110 / 110, 4 103, 2 100).
PowmShapeCost powm_shape_cost(int tpi, int limbs, int d) {
  const double rows = d ? (double)tpi * d : (double)tpi * limbs;
  const double alone = d ? std::max(155.0 + 8.0 * d, 21.5 * d) : std::max(100.0, 80.0 + 5.0 * limbs);
  const double full = d ? 38.0 + 17.5 * d : 10.0 + 13.5 * limbs;
  return PowmShapeCost{rows * alone, rows * full * tpi / 32.0};
}

// Two or three warps on a scheduler do not fill each other's gaps: 30 or, with the limb rows' carry chains, 35
// cycles a row more (measured / with them, two warps: 16 x 3 133 / 136, 16 x 6 245 / 246, 8 x 12 370 / 386).
double powm_shape_cycles(int tpi, int limbs, double groups, uint32_t sm_count, int digits) {
  const int d = digits < 0 ? powm_digits(tpi, limbs) : digits;
  const PowmShapeCost c = powm_shape_cost(tpi, limbs, d);
  double warps = groups * tpi / 32.0 / (4.0 * sm_count);  // a scheduler's, four a SM
  double gaps = 0;
  if (warps < 4.0) {
    warps = ceil(warps);  // the fullest scheduler sets the time
    if (warps > 1.0 && warps < 4.0) gaps = tpi * (d ? 30.0 * d : 35.0 * limbs);
  }
  return std::max(c.latency, c.work * 32.0 / tpi * warps + gaps);
}

bool powm_config_valid(const PowmConfig &c, uint32_t nlimbs) {
  if (c.window < 1 || c.window > 7) return false;
  if (c.dist == kDistDigit) return true;
  if (c.dist == kDistCta) return powm_cta_limbs(nlimbs) != 0 && (uint32_t)c.limbs == powm_cta_limbs(nlimbs);
  if ((uint64_t)c.tpi * c.limbs < nlimbs) return false;
  return powm_find(c.tpi, c.limbs) != nullptr;
}

PowmConfig powm_default_config(uint32_t nlimbs, uint32_t exp_bits, uint32_t count, xmpAlgorithm_t alg,
                               uint32_t sm_count, uint32_t want_cap) {
  PowmConfig best;
  if (alg == xmpAlgorithmDigitMP) {
    best.window = window_for_bits(exp_bits, false);
    best.dist = kDistDigit;
    return best;
  }
  // A score in limb multiply-adds, fitted before the digit kernels (powm_shape_cycles is their model).  Enough lanes
  // to give every SM a few warps; below that, spread instances wider.
  const double want_threads = (double)sm_count * 4 * 32;
  double best_score = 1e300;
  for (const auto &e : powm_registry()) {
    if (alg == xmpAlgorithmRegMP && e.tpi != 1) continue;
    if (alg == xmpAlgorithmDistributedMP && e.tpi == 1) continue;
    uint32_t cap = (uint32_t)e.tpi * e.limbs;
    if (cap < nlimbs || (want_cap && cap != want_cap)) continue;
    // Work per instance grows with capacity^2; lane overhead (shfl, carry
    // bookkeeping) is ~12 instructions per 4L multiply-adds.
    double pad = (double)cap / nlimbs;
    double work = pad * pad * (4.0 * e.limbs + (e.tpi > 1 ? 12.0 : 4.0)) / (4.0 * e.limbs);
    double threads = (double)count * e.tpi;
    double starve = threads < want_threads ? want_threads / threads : 1.0;
    double regs = e.limbs > 16 && e.tpi > 1 ? 1.5 : 1.0;  // register pressure beyond 16 limbs
    double score = work * starve * regs;
    if (score < best_score) {
      best_score = score;
      best.tpi = e.tpi;
      best.limbs = e.limbs;
    }
  }
  // Larger than every register kernel: the digit-serial kernel takes any size,
  // unless the caller forced a register distribution (then Unsupported).
  if (best.tpi == 0 && alg == xmpAlgorithmDefault) best.dist = kDistDigit;
  best.window = window_for_bits(exp_bits, best.dist != kDistDigit && powm_sliding(best.tpi, best.limbs));
  return best;
}

size_t powm_table_bytes(const PowmConfig &cfg, uint32_t nlimbs, uint32_t count, uint32_t cta_threads) {
  if (cfg.dist == kDistCta) return 0;  // the table is in shared memory
  if (cfg.dist == kDistDigit) {
    // table + N, x, b, m, r, r2 working arrays, all nlimbs+2 words per instance
    size_t words = ((size_t)1 << cfg.window) * nlimbs + 6 * ((size_t)nlimbs + 2);
    return words * 4 * round_up(count, 128);
  }
  size_t threads = round_up((uint32_t)std::min<uint64_t>((uint64_t)count * cfg.tpi, 0xffffff80ull), cta_threads);
  return threads * (size_t)powm_slot_words(cfg.tpi, cfg.limbs) *
         powm_table_entries(cfg.window, powm_sliding(cfg.tpi, cfg.limbs)) * 4;
}

xmpError_t powm_run(xmpHandle_t h, const PowmConfig &cfg0, const OutView &out, const ArrayView &base,
                    const ArrayView &exp, const ArrayView &mod, uint32_t count) {
  PowmConfig cfg = cfg0;
  if (cfg.dist == kDistDigit) return powm_digit_run(h, cfg, out, base, exp, mod, count);
  if (cfg.dist == kDistCta) {
    PowmArgs a;
    a.base = base;
    a.exp = exp;
    a.mod = mod;
    a.out = out;
    a.start = 0;
    a.count = count;
    a.window = cfg.window;
    a.table = nullptr;
    if (!powm_cta_launch((uint32_t)cfg.limbs, false, a, count, h->stream)) return xmpErrorUnsupported;
    return check_cuda();
  }
  const PowmKernelEntry *k = powm_find(cfg.tpi, cfg.limbs);
  if (!k) return xmpErrorUnsupported;
  size_t limit = scratch_limit(h);
  // Chunk so the window tables fit; shrink the window if even one CTA's instances do not fit, then the CTA
  // to one warp.
  int threads = 128;
  uint32_t per_block = 128 / cfg.tpi;
  uint32_t chunk = count;
  while (true) {
    size_t per_inst = (size_t)cfg.tpi * powm_slot_words(cfg.tpi, cfg.limbs) *
                      powm_table_entries(cfg.window, powm_sliding(cfg.tpi, cfg.limbs)) * 4;
    uint64_t fit = limit / per_inst;
    fit = fit / per_block * per_block;
    if (fit >= per_block) {
      chunk = (uint32_t)std::min<uint64_t>(count, fit);
      break;
    }
    if (cfg.window > 1) {
      cfg.window--;
    } else if (threads > 32) {
      threads = 32;
      per_block = 32 / cfg.tpi;
    } else {
      return xmpErrorIncreaseScratchLimit;
    }
  }
  xmpError_t e = ensure_scratch(h, powm_table_bytes(cfg, mod.nlimbs, chunk, threads));
  if (e != xmpErrorSuccess) return e;
  PowmArgs a;
  a.base = base;
  a.exp = exp;
  a.mod = mod;
  a.out = out;
  a.window = cfg.window;
  a.table = (uint32_t *)h->scratch;
  for (uint32_t start = 0; start < count; start += chunk) {
    a.start = start;
    a.count = std::min(chunk, count - start);
    k->launch(a, grid_for((uint64_t)a.count * cfg.tpi, threads), threads, h->stream);
  }
  return check_cuda();
}

}  // namespace xmpb

// Bytes of one warp's window-1 table, the least a lane kernel can run with.
static size_t powm_least_bytes(int tpi, int limbs) {
  return (size_t)32 * powm_slot_words(tpi, limbs) * powm_table_entries(1, powm_sliding(tpi, limbs)) * 4;
}

// Kernels chosen for their speed alone keep up to 20 digits a lane, 10 KB for one warp; where the scratch limit
// is below that, the kernel with the smallest tables that holds the precision takes their place.
static void powm_within_limit(PowmConfig &cfg, uint32_t nlimbs, size_t limit) {
  if (cfg.dist != kDistLanes || powm_least_bytes(cfg.tpi, cfg.limbs) <= limit) return;
  for (const auto &e : powm_registry()) {
    if ((uint32_t)(e.tpi * e.limbs) < nlimbs) continue;
    if (powm_least_bytes(e.tpi, e.limbs) >= powm_least_bytes(cfg.tpi, cfg.limbs)) continue;
    cfg.tpi = e.tpi;
    cfg.limbs = e.limbs;
  }
}

// The configuration for a problem shape under the handle's policy (default algorithm): a choice set
// for the exact shape, else one instance per CTA for small batches, else the selector, else the
// heuristic.  An explicit algorithm takes the heuristic restricted to it.
static PowmConfig powm_choose_config(xmpHandle_t h, uint32_t nlimbs, uint32_t exp_bits, uint32_t count) {
  PowmConfig cfg;
  const xmpAlgorithm_t alg = h->policy->algorithm;
  int src = 0;
  const bool tuned = (alg == xmpAlgorithmDefault) && tuner_lookup_powm(h, nlimbs, exp_bits, count, &cfg, &src);
  if (tuned && src == 1) return cfg;
  if (alg == xmpAlgorithmDefault && powm_cta_preferred(nlimbs, count, h->sm_count)) {
    cfg = PowmConfig();
    cfg.dist = kDistCta;
    cfg.limbs = (int)powm_cta_limbs(nlimbs);
    cfg.window = window_for_bits(exp_bits, true);
    return cfg;
  }
  if (!tuned) cfg = powm_default_config(nlimbs, exp_bits, count, alg, h->sm_count);
  if (alg == xmpAlgorithmDefault) powm_within_limit(cfg, nlimbs, scratch_limit(h));
  return cfg;
}

static xmpError_t powm_entry(xmpHandle_t h, xmpIntegers_t out, xmpIntegers_t base, xmpIntegers_t exp,
                             xmpIntegers_t mod, uint32_t count, const PowmConfig *forced) {
  if (!h || !out || !base || !exp || !mod) return xmpErrorInvalidParameter;
  int dev = h->device;
  if (out->device != dev || base->device != dev || exp->device != dev || mod->device != dev)
    return xmpErrorInvalidDevice;
  if (count == 0) return xmpErrorSuccess;
  DeviceGuard guard(dev);
  xmpExecutionPolicy_t p = h->policy;
  if (out->count < count) return xmpErrorInvalidCount;
  if (p->indices[0] && p->indices_count[0] < count) return xmpErrorInvalidCount;
  if (base->precision != out->precision || mod->precision != out->precision) return xmpErrorInvalidPrecision;

  PowmConfig cfg;
  if (forced) {
    cfg = *forced;
    if (cfg.dist == kDistCta) cfg.limbs = (int)powm_cta_limbs(mod->nlimbs);
  } else {
    cfg = powm_choose_config(h, mod->nlimbs, exp->precision, count);
  }
  if (!powm_config_valid(cfg, mod->nlimbs)) return xmpErrorUnsupported;

  bool aliased = (out == base || out == exp || out == mod);
  bool indexed = p->indices[0] || p->indices[1] || p->indices[2] || p->indices[3];
  OutTarget t;
  xmpError_t e = begin_output(h, out, aliased, indexed, &t);
  if (e != xmpErrorSuccess) return e;
  e = powm_run(h, cfg, view_out(out, t.limbs, p->indices[0]), view_in(base, p->indices[1], p->indices_count[1]),
               view_in(exp, p->indices[2], p->indices_count[2]), view_in(mod, p->indices[3], p->indices_count[3]),
               count);
  if (e != xmpErrorSuccess) return e;
  e = end_output(h, out, t);
  if (e != xmpErrorSuccess) return e;
  return check_cuda();
}

extern "C" {

xmpError_t XMPAPI xmpIntegersPowmAsync(xmpHandle_t h, xmpIntegers_t out, const xmpIntegers_t base,
                                        const xmpIntegers_t exp, const xmpIntegers_t mod, uint32_t count) {
  return powm_entry(h, out, base, exp, mod, count, nullptr);
}

xmpError_t XMPAPI xmpIntegersPowm(xmpHandle_t h, xmpIntegers_t out, const xmpIntegers_t base, const xmpIntegers_t exp,
                                   const xmpIntegers_t mod, uint32_t count) {
  xmpError_t e = xmpIntegersPowmAsync(h, out, base, exp, mod, count);
  if (e != xmpErrorSuccess) return e;
  DeviceGuard guard(h->device);
  cudaStreamSynchronize(h->stream);
  return check_cuda();
}

xmpError_t XMPAPI xmpIntegersPowmWithConfigAsync(xmpHandle_t h, xmpIntegers_t out, const xmpIntegers_t base,
                                                  const xmpIntegers_t exp, const xmpIntegers_t mod, uint32_t count,
                                                  const xmpPowmConfig_t *config) {
  if (!config) return xmpErrorInvalidParameter;
  PowmConfig c;
  c.dist = config->distribution;
  c.tpi = config->lanes;
  c.limbs = config->limbs;
  c.window = config->window;
  if (c.dist != kDistLanes && c.dist != kDistDigit && c.dist != kDistCta) return xmpErrorInvalidParameter;
  return powm_entry(h, out, base, exp, mod, count, &c);
}

xmpError_t XMPAPI xmpPowmKernelCount(int32_t *count) {
  if (!count) return xmpErrorInvalidParameter;
  *count = (int32_t)powm_registry().size();
  return xmpErrorSuccess;
}

xmpError_t XMPAPI xmpPowmKernelGet(int32_t index, int32_t *lanes, int32_t *limbs) {
  if (index < 0 || index >= (int32_t)powm_registry().size() || !lanes || !limbs) return xmpErrorInvalidParameter;
  *lanes = powm_registry()[index].tpi;
  *limbs = powm_registry()[index].limbs;
  return xmpErrorSuccess;
}

xmpError_t XMPAPI xmpPowmGetConfig(xmpHandle_t h, uint32_t precision, uint32_t exp_precision, uint32_t count,
                                   xmpPowmConfig_t *config) {
  if (!h || !config || precision == 0 || precision % 32 || exp_precision == 0 || exp_precision % 32)
    return xmpErrorInvalidParameter;
  const PowmConfig c = powm_choose_config(h, precision / 32, exp_precision, count);
  config->distribution = c.dist;
  config->lanes = c.tpi;
  config->limbs = c.limbs;
  config->window = c.window;
  return xmpErrorSuccess;
}

}  // extern "C"

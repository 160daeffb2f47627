// Integers spread over TPI lanes with L limbs each (lane g: limbs gL .. gL + L - 1): loads and stores
// between the interleaved arrays and the lanes' registers, shared by the powm, multiply and divide kernels.
#pragma once
#include "internal.h"
#include "mont.cuh"

namespace xmpb {

// Instance of a thread in a grid of TPI lanes each, formed in 64 bits: the threads of a batch that the device's
// memory holds pass 2^32 (33 to 48 limbs on 4 lanes: from 2^30 instances, a result of 155 GB).
template <int TPI>
__host__ __device__ __forceinline__ uint64_t lane_instance(uint32_t block, uint32_t threads, uint32_t thread) {
  return ((uint64_t)block * threads + thread) / TPI;
}

template <int TPI, int L>
__device__ __forceinline__ void load_lane_limbs(uint32_t (&x)[L], const uint32_t *limbs, uint32_t nlimbs,
                                                uint32_t stride, uint32_t e, uint32_t lane) {
  const uint32_t j0 = lane * L;
  if (L % 4 == 0) {
#pragma unroll
    for (int m = 0; m < L / 4; m++) {
      uint4 v = load_group(limbs, nlimbs, stride, e, j0 / 4 + m);
      x[4 * m] = v.x;
      x[4 * m + 1] = v.y;
      x[4 * m + 2] = v.z;
      x[4 * m + 3] = v.w;
    }
  } else {
#pragma unroll
    for (int k = 0; k < L; k++) x[k] = load_limb(limbs, nlimbs, stride, e, j0 + k);
  }
}

template <int TPI, int L>
__device__ __forceinline__ void store_lane_limbs(const uint32_t (&x)[L], uint32_t *limbs, uint32_t nlimbs,
                                                 uint32_t stride, uint32_t e, uint32_t lane) {
  const uint32_t j0 = lane * L;
  if (L % 4 == 0) {
#pragma unroll
    for (int m = 0; m < L / 4; m++) {
      uint32_t g = j0 / 4 + m;
      if (g * 4 < nlimbs) store_group(limbs, nlimbs, stride, e, g, make_uint4(x[4 * m], x[4 * m + 1], x[4 * m + 2], x[4 * m + 3]));
    }
  } else {
#pragma unroll
    for (int k = 0; k < L; k++)
      if (j0 + k < nlimbs) limb_ref(limbs, stride, e, j0 + k) = x[k];
  }
}

}  // namespace xmpb

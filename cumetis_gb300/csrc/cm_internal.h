// cm_internal.h -- declarations shared by the host and device translation
// units of libcm (not part of the public ABI).
#pragma once

#include <cstdarg>
#include <cstddef>
#include <cstdint>
#include <string>

#include "../../include/cm.h"

#ifdef __CUDACC__
#define CM_HOST_DEVICE __host__ __device__
#else
#define CM_HOST_DEVICE
#endif

// The default weight limit of a coarsening, (int)(1.5 * tvwgt / Coarsen_threshold)
// (cuMetis.cu:1828), at the ends of the int range where it lies beyond: the same
// for host and device, where a plain conversion need not be.
CM_HOST_DEVICE inline int32_t cm_weight_limit(int64_t tvwgt, int32_t coarsen_to) {
  const double x = 1.5 * (double)tvwgt / coarsen_to;
  return x >= (double)INT32_MAX ? INT32_MAX : x <= (double)INT32_MIN ? INT32_MIN : (int32_t)x;
}

// Reads a byte of every page of [p, p + bytes): an address that is not mapped ends
// the process here, on the host, before a kernel reads the array.
void cm_touch_pages(const void *p, size_t bytes);

// Records a formatted message for cm_last_error() and returns `code`.
int cm_fail(int code, const char *fmt, ...);

// Expanded-table dense convolution (axc_xtab.cu): route, scratch and launch.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "axc_internal.h"

namespace axc {

// What an expanded entry holds (table_form): two digits to the base 255, one byte, or nothing (only the exact products).
enum XtabMode { kXtabFull = 16, kXtabByte = 8, kXtabExact = 0, kXtabNone = -1 };

// Scratch bytes of the expanded-table route for this shape; 0 where the plan-based kernels serve the shape.
size_t xtab_scratch_bytes(const Geom &g);

int launch_xtab(const uint16_t *lut_dev, int mode, int centred, int e_min, const Geom &g, const Quant &q, const float *ranges_dev,
                const float *input, const float *filter, float *output, unsigned char *scratch, const axc_debug_out *dbg,
                const DeviceInfo &di, cudaStream_t stream);

}  // namespace axc

// Expanded-table dense convolution (axc_xtab.cu): route, scratch and launch.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "axc_internal.h"

namespace axc {

// What an expanded entry holds (table_form): two digits to the base 255, one byte, or nothing (only the exact products).  kXtabByte64: one byte, and the
// rows repeat every 64 activations.  kXtabRef: the entry itself, for the fp32 running total in K order.
enum XtabMode { kXtabRef = 17, kXtabFull = 16, kXtabByte = 8, kXtabByte64 = 9, kXtabExact = 0, kXtabNone = -1, kXtabAny = -2 };

// The fixed shared-window addresses of the dense kernels fit this device.
inline bool window_ok(const DeviceInfo &di) { return di.max_smem_optin >= 232448 && di.smem_base <= 2048u && di.smem_end >= 233472u; }

// Scratch bytes of the expanded-table route for this shape and a table kept as `mode` (kXtabAny: enough for every table); 0
// where the plan-based kernels serve the call.
size_t xtab_scratch_bytes(const Geom &g, int mode);
// Whether a call in the reference's order of additions is quicker on expanded tables.
bool xtab_ref_pays(const Geom &g);
// {pixels per tile, splits of K, tables from global memory} of a call that these kernels serve, on 148 SMs (diagnostics).
void xtab_config(const Geom &g, int mode, int32_t out3[3]);

// Operands of the quantised entry point and their zero points: the int32 result carries the terms
// K in_off f_off - f_off sum(a) - in_off sum(b); a tap outside the image has the code input_offset modulo 256.
struct QuantisedOperands {
    const uint8_t *input, *filter;
    int input_offset, filter_offset;
};

int launch_xtab(const uint16_t *lut_dev, int mode, int centred, int e_min, const Geom &g, const Quant &q, const float *ranges_dev,
                const float *input, const float *filter, float *output, unsigned char *scratch, const axc_debug_out *dbg,
                const DeviceInfo &di, cudaStream_t stream, const QuantisedOperands *u8 = nullptr);

}  // namespace axc

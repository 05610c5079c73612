// Quantisation parameters on the device, shared by the kernels that take ranges from device memory.
#pragma once
#include "axc_internal.h"
#include "axc_sched.h"

namespace axc {

// Range nudging on the device, operation by operation as on the host (axc_api.cu var_quant_props).
static __device__ __forceinline__ void dev_var_quant(float min_v, float max_v, float *scale, float *inv, float *offset)
{
    float s = 0.0f, i = 0.0f, nudged_min = 0.0f;
    if (min_v != 0.0f || max_v != 0.0f) {
        s = __fdiv_rn(__fsub_rn(max_v, min_v), 255.0f);
        const float zp_from_min = __fsub_rn(0.0f, __fdiv_rn(min_v, s));
        float zp;
        if (zp_from_min < 0.0f) zp = 0.0f;
        else if (zp_from_min > 255.0f) zp = 255.0f;
        else zp = roundf(zp_from_min);                       // half away from zero, like std::round
        nudged_min = __fmul_rn(__fsub_rn(0.0f, zp), s);      // a true subtraction: +0.0 for zp == 0
        i = __fdiv_rn(1.0f, s);
    }
    *scale = s; *inv = i; *offset = nudged_min;
}

static __device__ __forceinline__ DevQuant dev_quant_from_ranges(const float *__restrict__ ranges, int K)
{
    float s1, i1, o1, s2, i2, o2;
    dev_var_quant(ranges[0], ranges[1], &s1, &i1, &o1);
    dev_var_quant(ranges[2], ranges[3], &s2, &i2, &o2);
    DevQuant q;
    q.in_off = o1; q.in_inv = i1; q.f_off = o2; q.f_inv = i2;
    q.s1s2 = __fmul_rn(s1, s2); q.m1 = o1; q.m2 = o2;
    q.km1m2 = __fmul_rn(float(K), __fmul_rn(o1, o2));
    return q;
}

}  // namespace axc

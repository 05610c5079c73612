// Expanded-table dense convolution for sm_100a.
//
// Per K element a convolution looks the activations of its output pixels up in the table column of one weight per
// output channel.  For a group of channels and 8 consecutive K elements those columns are laid side by side in shared
// memory as an expanded table X[a][k][channel]: 256 rows of 8 x 16 bytes, where the 16 bytes at (a, k) are the entries of
// 8 channels (16-bit entries) or 16 channels (8-bit entries).  One LDS.128 per lane then returns 8 or 16 lookups, and
// since the 8 lanes of a quarter warp work on 8 different k, they read 8 different 16-byte bank groups whatever
// the activations are: every load is conflict-free and carries 128 useful bytes per clock.  The sums are taken by the
// tensor cores: the bytes of four lanes (four k of one pixel) are the A operand of an m16n8k32 u8 MMA against a constant
// matrix that adds the bytes of a channel into its accumulator.
//
// What is looked up (whole numbers throughout, so the total is the same):
//   8-bit entries    where the table differs from the exact product by values that span at most 255: that distance less its
//                    minimum.  The exact products are added by further MMAs on the codes themselves (one per 16 K elements,
//                    8 pixels and 16 channels).  Where that distance is the same for a and a + 64 the table has 64 rows.
//   16-bit entries   two digits to the base 255, so that one MMA with the weights 1 and 255 adds both into a single
//                    accumulator (256 does not fit a u8 operand; low and high bytes in accumulators of their own would
//                    halve the pixels a tile can hold).  A table that reaches past 65279 is stored less 128 (a + b) and its
//                    minimum; 128 times the sums of the activation and weight codes go back in at the end.
//   nothing          for an exact table: only the products.
//
// Bound: the shared-memory pipe, 64 lookups (16-bit) or 128 lookups (8-bit) per clock and SM, less what the expansion costs:
// 32 KiB read and 32 KiB written per 8 K elements and channel group, 512 clocks against one clock per pixel of the tile for the
// lookups - hence tiles of up to 2048 pixels, 3072 with two-digit entries and tables from global memory.  Measured on a B200:
// LDS.128 alone 4.02 clocks per warp instruction, LDS.128 + MMA 4.05 (the MMA pipe is half idle), against 4.50 with eight dp2a
// in the MMA's place.  A 16-bit lookup per lane and
// instruction (axc_sched.cu) cannot pass 32 per clock.
//
//   xprep_kernel   one pass over the input: 8-bit codes in pixel order (or the im2col rows where the channel count would
//                  waste a quarter of the 16-byte pieces), the patch sums of the dequantisation in the reference's order
//                  of additions; further blocks: quantised filter, transposed table, filter sums
//   xtab_kernel    the convolution; the transposed table (one row per weight) stays in shared memory
//   xfinal_kernel  only where K is split over CTAs: adds nothing, dequantises the integer sums
//
// Arithmetic (quantiser, table index, dequantisation) is the reference's, tf2/src/approx_nn_conv_kernels.cpp:167-296.
#include <cmath>

#include "axc_quant.cuh"
#include "axc_sched.h"
#include "axc_xtab.h"

namespace axc {

namespace {

// Shared window of a CTA (the host checks that it starts below 2 KiB and reaches 228 KiB):
//   [first byte, 3072)    barriers
//   [3072, 35840)         codes of the tile's pixels for 16 elements of K (exact table: four of them, up to 134144)
//   [35840, 65536)        transposed table, rows 0..57 (16-bit entries)
//   [65536, 131072)       two expanded tables, interleaved: row a of stage s at a*256 + s*128, so that an address is
//                         {offset in the row, a, 1, 0} and one byte permute puts the activation in
//   [131072, 232960)      transposed table, the other rows (8-bit entries: all 257 rows)
// 64 rows, two CTAs to an SM: codes [3072, 19456), transposed table [19456, 52352), tables of two chunks [65536, 98304), 64 rows of
// 256 bytes each, a chunk's two octets interleaved; the place in the ring is bit 6 of the row.
// With expanded tables from global memory: codes from 3072 up to 52224, tables of two chunks at 65536 and 131072, a chunk's
// two octets interleaved like the two stages above.
constexpr unsigned kCodes = 3072u;
constexpr unsigned kRowsLow = 35840u;
constexpr unsigned kTab = 65536u;
constexpr unsigned kRowsHigh = 131072u;
constexpr unsigned kWindowEnd = 233472u;
constexpr unsigned kRowsSmall = 19456u;        // rows that repeat every 64 activations: the transposed table
constexpr unsigned kWindowHalf = 98304u;       // and where the window ends, two CTAs to an SM
constexpr int kLowRows = 58;
constexpr int kWarps = 8;
constexpr int kNull = 256;                     // table row of a weight that does not exist: all zeros
static_assert(kRowsLow + kLowRows * 512u == kTab && kRowsHigh + (257u - kLowRows) * 512u <= kWindowEnd, "shared window");
constexpr int kWaitPolls = 1 << 20;
constexpr size_t kPartialMax = 64u << 20;      // integer sums of a call whose K is split over CTAs
constexpr double kXtabMinLookups = 8e6;        // (xtab_scratch_bytes)
constexpr size_t kXtMax = 640u << 20;          // expanded tables in global memory
constexpr int kModelSms = 148;                 // what the scratch size is computed for

// `n` bytes at `p` lie in the scratch of the call (debug flavour, as the checks of axc_internal.h)
#define AXC_SCRATCH_OK(P, p, n, site) \
    AXC_GLOBAL_OK(reinterpret_cast<const unsigned char *>(p) - reinterpret_cast<const unsigned char *>((P).hdr), (P).scratch_bytes - (long long)(n) + 1, site)

// ---- shared memory -----------------------------------------------------------------------------------------------
__device__ __forceinline__ uint4 lds128(unsigned addr)
{
    if (!AXC_SHARED_OK(addr, 16u, 0u, kWindowEnd, 301u)) return make_uint4(0, 0, 0, 0);
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}
__device__ __forceinline__ void sts64(unsigned addr, unsigned x, unsigned y)
{
    if (!AXC_SHARED_OK(addr, 8u, 0u, kWindowEnd, 306u)) return;
    asm volatile("st.shared.v2.u32 [%0], {%1,%2};" ::"r"(addr), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ unsigned lds32(unsigned addr)
{
    if (!AXC_SHARED_OK(addr, 4u, 0u, kWindowEnd, 302u)) return 0u;
    unsigned v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ void sts128(unsigned addr, uint4 v)
{
    if (!AXC_SHARED_OK(addr, 16u, 0u, kWindowEnd, 303u)) return;
    asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
// 16 bytes global -> shared, zeros where `bytes` is 0
__device__ __forceinline__ void cp_async16(unsigned dst, const void *src, unsigned bytes)
{
    if (!AXC_SHARED_OK(dst, 16u, 0u, kWindowEnd, 304u)) return;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_init(unsigned bar, unsigned count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
// `bytes` (a multiple of 16) global -> shared by the bulk copy engine, counted on `bar`
__device__ __forceinline__ void bulk_copy(unsigned dst, const void *src, unsigned bytes, unsigned bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Polls after which a wait gives up, about a second.  The debug flavour reads them from device memory, so that a test can make
// the waits of one kernel run out: {xexpand_kernel, xtab_kernel}.
#ifdef AXC_BOUNDS_CHECK
__device__ int g_wait_polls[2] = {kWaitPolls, kWaitPolls};
#define AXC_WAIT_POLLS(kernel) (*(volatile int *)&g_wait_polls[kernel])
#else
#define AXC_WAIT_POLLS(kernel) kWaitPolls
#endif
// Waits for the phase `parity`; gives up after `polls` (`ok` stays false from then on, later waits return at once).
// A kernel whose wait gave up starts no further copy, finishes with whatever is in shared memory (every address is in bounds
// whatever the tables hold), waits for its own copies in flight and leaves 3 in the header's status.
__device__ __forceinline__ void mbar_wait(unsigned bar, unsigned parity, bool &ok, int polls)
{
#ifdef AXC_BOUNDS_CHECK
    if (polls <= 0) ok = false;
#endif
    for (int it = 0; ok; ++it) {
        unsigned done;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(done) : "r"(bar), "r"(parity) : "memory");
        if (done) return;
        if (it >= polls) ok = false;
    }
}
// The end of a kernel that gave up: the phase that a copy in flight completes.
__device__ __forceinline__ void mbar_drain(unsigned bar, unsigned parity)
{
    bool ok = true;
    mbar_wait(bar, parity, ok, kWaitPolls);
}

// Programmatic dependent launch: the kernels of a call after the first are launched so that each may start while the one before it
// runs.  pdl_trigger: the next kernel may be brought in; pdl_wait: everything before this kernel is complete and visible.
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <unsigned SEL>
__device__ __forceinline__ unsigned prmt(unsigned a, unsigned b)
{
    unsigned d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "n"(SEL));
    return d;
}
__device__ __forceinline__ unsigned prmt_r(unsigned a, unsigned b, unsigned sel)
{
    unsigned d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
    return d;
}
__device__ __forceinline__ void mma_k32(int (&c)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0, unsigned b1)
{
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.u8.s32 {%0,%1,%2,%3},{%4,%5,%6,%7},{%8,%9},{%0,%1,%2,%3};"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// The 8-bit code of x: trunc((x - off) * inv + 0.5) with three separately rounded operations
// (tf2/src/approx_nn_conv_kernels.cpp:293), clamped to 0..255, NaN -> 0.  Adding 2^23 with rounding towards minus infinity
// leaves the integer part in the low mantissa bits: full-rate instructions in place of a conversion.
__device__ __forceinline__ unsigned code_of(float x, float off, float inv)
{
    const float v = __fadd_rn(__fmul_rn(__fsub_rn(x, off), inv), 0.5f);
    return __float_as_uint(__fadd_rd(fminf(fmaxf(v, 0.0f), 255.0f), 8388608.0f)) & 0xFFu;
}

// The codes of four neighbouring values as a word.
__device__ __forceinline__ unsigned codes_of(const float4 &x, float off, float inv)
{
    auto biased = [&](float y) {
        const float v = __fadd_rn(__fmul_rn(__fsub_rn(y, off), inv), 0.5f);
        return __float_as_uint(__fadd_rd(fminf(fmaxf(v, 0.0f), 255.0f), 8388608.0f));
    };
    return prmt<0x5410>(prmt<0x0040>(biased(x.x), biased(x.y)), prmt<0x0040>(biased(x.z), biased(x.w)));
}

// ------------------------------------------------------------------------------------------------------------------
// preparation
// ------------------------------------------------------------------------------------------------------------------
struct XGeom {
    int N, H, W, C, KH, KW, Cout, sh, sw, dh, dw, ph, pw, OH, OW, K, M;
    int CC;             // 16-byte pieces of codes per pixel (im2col: per output pixel)
    int chunks;         // 16-element steps of K: KH*KW*CC, or CC with im2col
    int im2col;
    int TNC;            // channels per tile: 8 (16-bit entries) or 16
    int tiles_n;
};

constexpr int kPrepThreads = 512;

struct PrepParams {
    XGeom g;
    const float *input, *filter;
    const uint8_t *input_u8, *filter_u8;      // quantised operands (then the fp32 pointers are NULL): the code c counts as c - pad
    int pad;                                  // resp. c, which the call's ranges map back to c
    const uint16_t *lut;
    const float *ranges;
    DevQuant host_q;
    float in_floor;
    int mode, centred, e_min;
    int *acode, *bcode;         // sums of activation / weight codes where the end of the call needs them, else NULL
    uint4 *zeros;               // integer sums of a call whose K is split, to be set to zero: 16-byte pieces of them, or NULL
    long long zero_pieces;
    unsigned char *codes, *tt;
    uint16_t *wrow;
    uint2 *wb;
    float *asum, *bsum;
    uint8_t *qf_debug;
    PlanHeader *hdr;
    long long scratch_bytes;
    int blocks_sum, blocks_w, blocks_t;      // first blocks, last but one and last; the rest are input tiles
    int TH, TW, tiles_y, tiles_x, RH, RW, pitch, vec;
    int sums;                                 // patch and filter sums are asked for (a quantised call has none)
    int bytes_at, bytes_pitch;                // im2col: codes of the staged taps behind the taps (-1: none), bytes per region row
};

__host__ __device__ __forceinline__ bool two_bytes(int mode) { return mode == kXtabFull || mode == kXtabRef; }

// channel of slot s in a piece: the order in which a lane's accumulators hold four neighbouring channels
__device__ __forceinline__ int slot_channel(int mode, int s)
{
    if (two_bytes(mode)) return s;
    return ((s >> 3) << 3) + ((s >> 1) & 1) * 4 + ((s >> 2) & 1) * 2 + (s & 1);     // 0 1 4 5 2 3 6 7 8 9 12 13 10 11 14 15
}

// shared-memory address of a row of the transposed table
__device__ __forceinline__ unsigned row_address(int mode, unsigned row)
{
    if (mode == kXtabByte64) return kRowsSmall + row * 128u;
    if (!two_bytes(mode)) return kRowsHigh + row * 256u;
    return row < unsigned(kLowRows) ? kRowsLow + row * 512u : kRowsHigh + (row - kLowRows) * 512u;
}

// (The operands' type is a template parameter of the preparation: a branch on it between loads has each of them waited for before
// the next is issued - 53 us instead of 13 for the sums of a filter with K = 4608.)
template <bool U8>
__device__ __forceinline__ float filter_value(const XGeom &g, const float *f, const uint8_t *u8, size_t at)
{
    if (!AXC_GLOBAL_OK((long long)at, (long long)g.K * g.Cout, 320u)) return 0.0f;
    return U8 ? float(__ldg(u8 + at)) : __ldg(f + at);
}

__device__ __forceinline__ bool staged_ok(long long at, int count, unsigned site)      // floats of xprep_kernel's shared memory
{
#ifdef AXC_BOUNDS_CHECK
    unsigned size;
    asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(size));
    return AXC_GLOBAL_OK(at, (long long)(size / 4) - count + 1, site);
#else
    return true;
#endif
}

// K index of element i of chunk ch, or -1 where there is none
__device__ __forceinline__ int k_of(const XGeom &g, int ch, int i)
{
    if (g.im2col) {
        const int k = ch * 16 + i;
        return k < g.K ? k : -1;
    }
    const int tap = ch / g.CC, c = (ch - tap * g.CC) * 16 + i;
    return c < g.C ? tap * g.C + c : -1;
}

// Filter sums in l order (tf2/src/approx_nn_conv_kernels.cpp:187-197), 32 channels per block.  Bound by the order: a chain of K
// additions per channel, 4 clocks each.  One warp adds, a lane per channel, and does nothing else: eight others have the rows
// brought into a ring of six stages of 64 (cp.async).  The whole preparation of 3x3 512 -> 512 at 7x7, one image: 28 us; with the rows
// staged through registers by the whole block, 256 at a time between barriers, 40; asked for by the adding warp itself 104; by a
// bulk copy per row 143.  The sums of the codes, where they are asked for, are the other warps'.
constexpr int kSumRows = 64, kSumStages = 6, kSumLoaders = 256;
constexpr size_t kSumSmem = size_t(kSumRows) * kSumStages * 128 + 128 + 128;      // the ring, code sums, barriers

template <bool U8>
__device__ void prep_filter_sums(const PrepParams &P, const DevQuant &q, int block, float *stage)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int j = block * 32 + lane, K = P.g.K, Cout = P.g.Cout;
    const bool have = j < Cout;
    const unsigned ring = (unsigned)__cvta_generic_to_shared(stage), full = ring + kSumRows * kSumStages * 128u + 128u, empty = full + 8u * kSumStages;
    if (P.sums) {
        if (threadIdx.x == 0) {
            for (int s = 0; s < kSumStages; ++s) { mbar_init(full + 8u * s, kSumLoaders); mbar_init(empty + 8u * s, 1); }
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        }
        __syncthreads();
    }
    bool ok = true;
    const int stages = (K + kSumRows - 1) / kSumRows;
    if (P.sums && warp == 0) {
        float acc = 0.0f;
        for (int i = 0; i < stages; ++i) {
            const int at = i % kSumStages, n = min(kSumRows, K - i * kSumRows);
            mbar_wait(full + 8u * at, (i / kSumStages) & 1, ok, kWaitPolls);
            const float *src = stage + at * (kSumRows * 32) + lane;
            float u[2][16];
            auto rows16 = [&](int l, float (&to)[16]) {
#pragma unroll
                for (int e = 0; e < 16; ++e) to[e] = src[(l + e) * 32];
            };
            auto add16 = [&](const float (&a)[16]) {
#pragma unroll
                for (int e = 0; e < 16; ++e) acc = __fadd_rn(acc, a[e]);
            };
            if (n == kSumRows) {                                   // the next 16 rows are read while the last 16 are added
                rows16(0, u[0]); rows16(16, u[1]);
                add16(u[0]); rows16(32, u[0]);
                add16(u[1]); rows16(48, u[1]);
                add16(u[0]); add16(u[1]);
            } else
                for (int l = 0; l < n; ++l) acc = __fadd_rn(acc, src[l * 32]);
            __syncwarp();
            if (lane == 0) mbar_arrive(empty + 8u * at);
        }
        if (have && AXC_SCRATCH_OK(P, P.bsum + j, 4, 322u)) P.bsum[j] = acc;
    } else if (P.sums && warp <= kSumLoaders / 32) {
        const int who = int(threadIdx.x) - 32, wide = (Cout & 3) == 0 && (reinterpret_cast<uintptr_t>(P.filter) & 15u) == 0 ? 1 : 0;
        for (int i = 0; i < stages; ++i) {
            const int at = i % kSumStages, l0 = i * kSumRows;
            if (i >= kSumStages) mbar_wait(empty + 8u * at, (i / kSumStages - 1) & 1, ok, kWaitPolls);
            if (!ok) break;
            const unsigned to = ring + unsigned(at) * (kSumRows * 128u);
            if (wide) {                                            // 16 bytes at a time, 8 pieces to a row
#pragma unroll
                for (int e = 0; e < kSumRows * 8 / kSumLoaders; ++e) {
                    const int x = e * kSumLoaders + who, l = l0 + (x >> 3), c = block * 32 + (x & 7) * 4;
                    if (l < K && c < Cout && AXC_GLOBAL_OK((long long)l * Cout + c + 3, (long long)K * Cout, 320u)) cp_async16(to + unsigned(x) * 16u, P.filter + (size_t)l * Cout + c, 16u);
                }
            } else {
#pragma unroll
                for (int e = 0; e < kSumRows * 32 / kSumLoaders; ++e) {
                    const int x = e * kSumLoaders + who, l = l0 + (x >> 5), c = block * 32 + (x & 31);
                    if (l < K && c < Cout && AXC_GLOBAL_OK((long long)l * Cout + c, (long long)K * Cout, 319u))
                        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(to + unsigned(x) * 4u), "l"(P.filter + (size_t)l * Cout + c) : "memory");
                }
            }
            // the barrier hears of it when this thread's copies have arrived
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(full + 8u * at) : "memory");
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    }
    if (!ok) atomicExch(&P.hdr->status, 3);
    if (P.bcode) {
        // the warps after the loaders share the rows
        int *sums = reinterpret_cast<int *>(stage) + kSumRows * kSumStages * 32;
        constexpr int kFirst = kSumLoaders / 32 + 1, kStep = kPrepThreads / 32 - kFirst;
        if (warp == kFirst) sums[lane] = 0;
        __syncthreads();
        int codes = 0;
        if (warp >= kFirst)
            for (int l0 = warp - kFirst; l0 < K; l0 += 8 * kStep) {
                float v[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) v[e] = have && l0 + e * kStep < K ? filter_value<U8>(P.g, P.filter, P.filter_u8, (size_t)(l0 + e * kStep) * Cout + j) : 0.0f;
#pragma unroll
                for (int e = 0; e < 8; ++e) codes += have && l0 + e * kStep < K ? int(code_of(v[e], q.f_off, q.f_inv)) : 0;
            }
        if (warp >= kFirst) atomicAdd(sums + lane, codes);
        __syncthreads();
        if (warp == kFirst && have && AXC_SCRATCH_OK(P, P.bcode + j, 4, 323u)) P.bcode[j] = sums[lane];
    }
}

template <bool U8>
__global__ void __launch_bounds__(kPrepThreads, 2) xprep_kernel(const PrepParams P)
{
    extern __shared__ __align__(16) float prep_smem[];
    pdl_trigger();
    const XGeom &g = P.g;
    const int tid = threadIdx.x;
    if (P.zeros)
        for (long long x = (long long)blockIdx.x * kPrepThreads + tid; x < P.zero_pieces; x += (long long)gridDim.x * kPrepThreads)
            if (AXC_SCRATCH_OK(P, P.zeros + x, 16, 345u)) P.zeros[x] = make_uint4(0, 0, 0, 0);
    const DevQuant q = P.ranges ? dev_quant_from_ranges(P.ranges, g.K) : P.host_q;
    int b = int(blockIdx.x);
    if (b == 0 && tid == 0) {
        // header: the parameters of the call; every lookup is one conflict-free step, no plan to rebuild
        *reinterpret_cast<DevQuant *>(reinterpret_cast<unsigned char *>(P.hdr) + kDevQuantOffset) = q;
        P.hdr->magic = kXtabMagic;
        P.hdr->dirty = 0; P.hdr->fallback = 0; P.hdr->status = 0;
    }
    if (b < P.blocks_sum) {
        prep_filter_sums<U8>(P, q, b, prep_smem);
        return;
    }
    // sums of filter and patches first: their chains of additions are the longest work of a block
    b -= P.blocks_sum;
    const int tiles = int(gridDim.x) - P.blocks_sum - P.blocks_w - P.blocks_t;
    const unsigned z = code_of(0.0f, q.in_off, q.in_inv);        // code of a tap outside the image; codes are stored xor z
    if (b >= tiles && b < tiles + P.blocks_w) {
        b -= tiles;
        // wrow[tile][chunk][octet][k][slot]: where the table row of the slot's weight lies, in 16-byte units; wb[tile][chunk][lane]:
        // the weight codes as B operand of the exact products.  A warp takes a chunk at a time, eight weights (four of two-digit
        // entries) per lane: all loads of a chunk are in flight together and nothing is divided per weight.
        const int lane = tid & 31;
        const long long total = (long long)g.tiles_n * g.chunks;
        for (long long tc = (long long)b * (kPrepThreads / 32) + (tid >> 5); tc < total; tc += (long long)P.blocks_w * (kPrepThreads / 32)) {
            const int nt = int(tc / g.chunks), ch = int(tc - (long long)nt * g.chunks);
            const int slot = lane & (g.TNC - 1), cj = slot_channel(P.mode, slot), j = nt * g.TNC + cj;
            const bool full = two_bytes(P.mode);
            float v[8];
            int k[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const int kk = full ? e * 4 + (lane >> 3) : (lane >> 4) * 8 + e;     // octet * 8 + t + 4p
                const int i = P.mode == kXtabRef ? kk : ((kk & 3) << 2) + ((kk >> 3) << 1) + ((kk >> 2) & 1);   // element 4t + 2*octet + p
                k[e] = (!full || e < 4) && j < g.Cout ? k_of(g, ch, i) : -1;
                v[e] = k[e] >= 0 ? filter_value<U8>(g, P.filter, P.filter_u8, (size_t)k[e] * g.Cout + j) : 0.0f;
            }
            unsigned row[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                if (full && e >= 4) break;
                row[e] = kNull;
                if (k[e] >= 0) {
                    row[e] = code_of(v[e], q.f_off, q.f_inv);
                    if (P.qf_debug) P.qf_debug[(size_t)k[e] * g.Cout + j] = uint8_t(row[e]);
                }
                const int kk = full ? e * 4 + (lane >> 3) : (lane >> 4) * 8 + e;
                uint16_t *w = P.wrow + tc * (16 * g.TNC) + kk * g.TNC + slot;
                if (P.mode != kXtabExact && AXC_SCRATCH_OK(P, w, 2, 324u)) *w = uint16_t(row_address(P.mode, row[e]) >> 4);
            }
            if (!full) {
                // B operand half h, column n: channel (n>>1)*4 + 2h + (n&1); lane (n, t) holds elements 4t..4t+3, of which this
                // lane has 2*octet and the one after it
                const int h = (cj >> 1) & 1, n = (cj >> 2) * 2 + (cj & 1);
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    unsigned char *w = reinterpret_cast<unsigned char *>(P.wb + tc * 32 + n * 4 + t) + h * 4 + 2 * (lane >> 4);
                    if (AXC_SCRATCH_OK(P, w, 2, 325u)) *reinterpret_cast<uint16_t *>(w) = uint16_t((row[t] & 0xFFu) | (row[4 + t] & 0xFFu) << 8);   // kNull: 0
                }
            }
        }
        return;
    }
    if (b >= tiles) {
        b -= tiles + P.blocks_w;
        // transposed table: row = weight, column = stored code; row 256 = zeros
        const int row_shift = P.mode == kXtabByte64 ? 7 : 8;       // (64 entries, twice)
        const int total = 257 << row_shift;
        for (int x = b * kPrepThreads + tid; x < total; x += P.blocks_t * kPrepThreads) {
            const int w = x >> row_shift, a = (x & ((1 << row_shift) - 1)) ^ int(z);
            const int less = (P.mode == kXtabFull ? 128 * (a + w) * P.centred : a * w) + P.e_min;
            const int v = w < 256 ? int(__ldg(P.lut + a * 256 + w)) - less : 0;
            if (!AXC_SCRATCH_OK(P, P.tt + x * (two_bytes(P.mode) ? 2 : 1), two_bytes(P.mode) ? 2 : 1, 326u)) continue;
            if (P.mode == kXtabRef) reinterpret_cast<uint16_t *>(P.tt)[x] = w < 256 ? __ldg(P.lut + a * 256 + w) : 0;
            else if (P.mode == kXtabFull) reinterpret_cast<uint16_t *>(P.tt)[x] = uint16_t(v % 255 + (v / 255) * 256);
            else P.tt[x] = (unsigned char)v;
        }
        return;
    }

    // ---- an input tile: TH x TW output pixels of one image, the taps they read staged in shared memory ----------------
    // Bound by memory where K is short, by the additions' order where it is long: a pixel's sum is a chain of K dependent
    // additions (4 clocks each), so the host takes tiles that put as many pixels as possible on the chip at once (prep_tile).
    const int tx = b % P.tiles_x, rest = b / P.tiles_x;
    const int ty = rest % P.tiles_y, n = rest / P.tiles_y;
    const int oy0 = ty * P.TH, ox0 = tx * P.TW;
    const int iy0 = oy0 * g.sh - g.ph, ix0 = ox0 * g.sw - g.pw;
    // codes of the region's input pixels are written by the tile whose region starts closest before them
    const int own_h = ty + 1 < P.tiles_y ? P.TH * g.sh : P.RH, own_w = tx + 1 < P.tiles_x ? P.TW * g.sw : P.RW;
    const unsigned zz = z * 0x01010101u;
    // codes[piece][pixel][16]: the pieces of neighbouring pixels lie side by side, so that the producers read whole lines
    const int planes = g.N * g.H * g.W, region = P.RH * P.RW;
    // the sum of the codes of every staged pixel (z for one outside the image) behind the staged taps, where it is asked for
    int *pix_codes = reinterpret_cast<int *>(prep_smem + region * P.pitch);
    unsigned char *const code_bytes = reinterpret_cast<unsigned char *>(prep_smem) + P.bytes_at;
    if (P.vec) {
        // Eight lanes read 128 bytes of a pixel, a warp four pixels: whole sectors in, and 64-byte runs of codes out.  A thread keeps
        // where its pixel's piece comes from and goes to, and steps along the channels (140 instructions per piece otherwise, twice
        // what is left; the loop is bound by them).
        const int C4 = g.C >> 2;
        int lp = 1;
        while (lp < C4 && lp < 8) lp <<= 1;                       // lanes per pixel
        const int px_step = kPrepThreads / lp, c_lane = tid & (lp - 1), c_blocks = (C4 + lp - 1) / lp, code_step = lp * planes;
        const int p = tid / lp;
        int ry = p / P.RW, rx = p - ry * P.RW, cb = 0;
        const int step_y = px_step / P.RW, step_x = px_step - step_y * P.RW;
        int from = -1, at = -1, code_to = -1;                     // float4 of the input, float of the stage, word of the codes; -1: none
        auto pixel = [&]() {
            from = at = code_to = -1;
            if (ry >= P.RH || c_lane >= C4) return;
            const int iy = iy0 + ry, ix = ix0 + rx;
            at = (ry * P.RW + rx) * P.pitch + c_lane * 4;
            if (unsigned(iy) < unsigned(g.H) && unsigned(ix) < unsigned(g.W)) {
                const int pix = (n * g.H + iy) * g.W + ix;
                from = pix * C4 + c_lane;
                if (ry < own_h && rx < own_w) code_to = ((c_lane >> 2) * planes + pix) * 4 + (c_lane & 3);
            }
        };
        pixel();
        constexpr int kBatch = 4;                                 // loads of a thread in flight
        int sum = 0, cb_done = 0, done = p;                       // code sum of the pixel being finished
        for (int left = (region + px_step - 1) / px_step * c_blocks; left > 0; left -= kBatch) {
            float4 v[kBatch];
            int to[kBatch], code_at[kBatch];
#pragma unroll
            for (int u = 0; u < kBatch; ++u) {
                v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                const bool in_c = cb * lp + c_lane < C4;
                to[u] = in_c ? at : -1;
                code_at[u] = in_c ? code_to : -1;
                if (from >= 0 && in_c && AXC_GLOBAL_OK((long long)from, (long long)planes * C4, 328u)) {
                    if (U8) {
                        const uchar4 w = __ldg(reinterpret_cast<const uchar4 *>(P.input_u8) + from);
                        v[u] = make_float4(float(int(w.x) - P.pad), float(int(w.y) - P.pad), float(int(w.z) - P.pad), float(int(w.w) - P.pad));
                    } else v[u] = __ldg(reinterpret_cast<const float4 *>(P.input) + from);
                }
                if (++cb == c_blocks) {
                    cb = 0;
                    rx += step_x; ry += step_y;
                    if (rx >= P.RW) { rx -= P.RW; ++ry; }
                    pixel();
                } else {
                    if (from >= 0) from += lp;
                    if (code_to >= 0) code_to += code_step;
                    if (at >= 0) at += lp * 4;
                }
            }
#pragma unroll
            for (int u = 0; u < kBatch; ++u) {
                v[u].x = max_keep_nan(v[u].x, P.in_floor); v[u].y = max_keep_nan(v[u].y, P.in_floor);
                v[u].z = max_keep_nan(v[u].z, P.in_floor); v[u].w = max_keep_nan(v[u].w, P.in_floor);
                if (P.sums && to[u] >= 0 && staged_ok(to[u], 4, 329u)) *reinterpret_cast<float4 *>(prep_smem + to[u]) = v[u];
                if (code_at[u] >= 0 || P.acode) {
                    const unsigned w = codes_of(v[u], q.in_off, q.in_inv);
                    if (code_at[u] >= 0 && AXC_SCRATCH_OK(P, P.codes + (size_t)(unsigned)code_at[u] * 4, 4, 330u)) reinterpret_cast<unsigned *>(P.codes)[(unsigned)code_at[u]] = w ^ zz;
                    if (P.acode) {                                // (the same for all threads)
                        if (to[u] >= 0) sum = int(__dp4a(w, 0x01010101u, unsigned(sum)));
                        if (++cb_done == c_blocks) {
                            for (int d = lp >> 1; d > 0; d >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, d);
                            if (c_lane == 0 && done < region && staged_ok(region * P.pitch + done, 1, 331u)) pix_codes[done] = sum;
                            sum = cb_done = 0;
                            done += px_step;
                        }
                    }
                }
            }
        }
    } else {
        // The taps of a region row lie side by side in memory: a warp takes 256 of them at a time, eight loads in flight per lane.
        if (P.acode && !g.im2col) {
            for (int x = tid; x < region; x += kPrepThreads)
                if (staged_ok(region * P.pitch + x, 1, 327u)) pix_codes[x] = 0;
        }
        const int row = P.RW * g.C, parts = (row + 255) >> 8, lane = tid & 31;
        const int x_lo = ix0 * g.C, x_end = g.W * g.C;
        const unsigned per_c = g.C > 1 ? 0xFFFFFFFFu / unsigned(g.C) + 1u : 0u;       // e / C for e * C < 2^32
        for (int task = tid >> 5; task < P.RH * parts; task += kPrepThreads / 32) {
            const int ry = task / parts, e0 = (task - ry * parts) * 256 + lane, iy = iy0 + ry;
            const bool row_in = unsigned(iy) < unsigned(g.H);
            const long long base = ((long long)n * g.H + iy) * x_end + x_lo;
            float v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int e = e0 + u * 32;
                const bool in = row_in && e < row && unsigned(x_lo + e) < unsigned(x_end) && AXC_GLOBAL_OK(base + e, (long long)planes * g.C, 332u);
                v[u] = !in ? 0.0f : U8 ? float(int(__ldg(P.input_u8 + base + e)) - P.pad) : __ldg(P.input + base + e);
            }
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int e = e0 + u * 32;
                if (e >= row) break;
                v[u] = max_keep_nan(v[u], P.in_floor);
                const int at = ry * P.RW * P.pitch + e + (P.pitch != g.C ? int(__umulhi(unsigned(e), per_c)) : 0);
                if (staged_ok(at, 1, 333u)) prep_smem[at] = v[u];
                if (P.bytes_at >= 0 && staged_ok(P.bytes_at / 4 + (ry * P.bytes_pitch + e) / 4, 1, 334u)) code_bytes[ry * P.bytes_pitch + e] = (unsigned char)code_of(v[u], q.in_off, q.in_inv);
            }
        }
        if (!g.im2col) {
            // codes: a piece of a pixel per thread, neighbouring pixels side by side
            __syncthreads();
            for (int x = tid; x < region * g.CC; x += kPrepThreads) {
                const int piece = x / region, local = x - piece * region, ry = local / P.RW, rx = local - ry * P.RW;
                const int iy = iy0 + ry, ix = ix0 + rx;
                const bool mine = unsigned(iy) < unsigned(g.H) && unsigned(ix) < unsigned(g.W) && ry < own_h && rx < own_w;
                if (!mine && !P.acode) continue;
                const float *src = prep_smem + local * P.pitch + piece * 16;
                const int count = min(16, g.C - piece * 16);
                if (!staged_ok(src - prep_smem, count, 335u)) continue;
                unsigned w[4] = {0, 0, 0, 0};
#pragma unroll
                for (int e = 0; e < 16; ++e)
                    if (e < count) w[e >> 2] |= code_of(src[e], q.in_off, q.in_inv) << (8 * (e & 3));
                if (P.acode && staged_ok(region * P.pitch + local, 1, 342u))
                    atomicAdd(pix_codes + local, int(__dp4a(w[0], 0x01010101u, __dp4a(w[1], 0x01010101u, __dp4a(w[2], 0x01010101u, __dp4a(w[3], 0x01010101u, 0u))))));
                uint4 *dst = reinterpret_cast<uint4 *>(P.codes) + ((size_t)piece * planes + ((size_t)n * g.H + iy) * g.W + ix);
                if (mine && AXC_SCRATCH_OK(P, dst, 16, 343u)) *dst = make_uint4(w[0] ^ zz, w[1] ^ zz, w[2] ^ zz, w[3] ^ zz);
            }
        }
    }
    __syncthreads();
    // patch sums (tf2/src/approx_nn_conv_kernels.cpp:272-295): the raw taps in K order, one thread per output pixel
    const int run = g.dw == 1 ? g.KW * g.C : g.C, runs_x = g.dw == 1 ? 1 : g.KW;      // taps that lie side by side (no padding between pixels)
    for (int o = tid; o < P.TH * P.TW; o += kPrepThreads) {
        const int ly = o / P.TW, lx = o - ly * P.TW;
        const int oy = oy0 + ly, ox = ox0 + lx;
        if (oy >= g.OH || ox >= g.OW) continue;
        const long long m = ((long long)n * g.OH + oy) * g.OW + ox;
        const int first = ly * g.sh * P.RW + lx * g.sw;            // region pixel of the first tap
        float s = 0.0f;
        int codes = 0;
        if (!g.im2col && P.acode)
            for (int ky = 0; ky < g.KH; ++ky)
                for (int kx = 0; kx < g.KW; ++kx) codes += pix_codes[first + ky * g.dh * P.RW + kx * g.dw];
        if (P.sums && P.vec && (g.C & 15) == 0) {
            // 16 channels at a time over all taps, the next ones on their way while the last ones are added
            const int steps = g.KH * g.KW * (g.C >> 4);
            const float *src = prep_smem + first * P.pitch;
            int c = 0, kx = 0;
            float4 v[2][4];
            auto take = [&](float4 (&to)[4]) {
                if (!staged_ok(src - prep_smem, 16, 336u)) return;
#pragma unroll
                for (int e = 0; e < 4; ++e) to[e] = reinterpret_cast<const float4 *>(src)[e];
                src += 16; c += 16;
                if (c == g.C) {
                    c = 0;
                    src += g.dw * P.pitch - g.C;
                    if (++kx == g.KW) { kx = 0; src += (g.dh * P.RW - g.KW * g.dw) * P.pitch; }
                }
            };
            auto add = [&](const float4 (&a)[4]) {
#pragma unroll
                for (int e = 0; e < 4; ++e) s = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(s, a[e].x), a[e].y), a[e].z), a[e].w);
            };
            take(v[0]);
            int i = 1;
            for (; i + 1 < steps; i += 2) {
                take(v[1]);
                add(v[0]);
                take(v[0]);
                add(v[1]);
            }
            if (i < steps) {
                take(v[1]);
                add(v[0]);
                add(v[1]);
            } else add(v[0]);
        } else if (P.sums && P.vec) {
            for (int ky = 0; ky < g.KH; ++ky)
                for (int kx = 0; kx < g.KW; ++kx) {
                    const float *src = prep_smem + (first + ky * g.dh * P.RW + kx * g.dw) * P.pitch;
                    if (!staged_ok(src - prep_smem, g.C, 337u)) continue;
#pragma unroll 4
                    for (int c = 0; c < g.C; c += 4) {
                        const float4 v = *reinterpret_cast<const float4 *>(src + c);
                        s = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(s, v.x), v.y), v.z), v.w);
                    }
                }
        } else if (P.sums) {
            const bool joined = P.pitch == g.C;                   // a run crosses pixels only where they lie side by side
            const int len = joined ? run : g.C, xs = joined ? runs_x : g.KW;
            for (int ky = 0; ky < g.KH; ++ky)
                for (int kx = 0; kx < xs; ++kx) {
                    const float *src = prep_smem + (first + ky * g.dh * P.RW + kx * g.dw) * P.pitch;
                    if (!staged_ok(src - prep_smem, len, 338u)) continue;
#pragma unroll 8
                    for (int c = 0; c < len; ++c) s = __fadd_rn(s, src[c]);
                }
        }
        if (g.im2col) {
            // im2col rows of codes off the runs of taps that lie side by side in a region row, a word at a time: one aligned word read,
            // one shift to the run's start, one to the place in the row (every word put together byte by byte: 25 instructions)
            uint4 *dst = reinterpret_cast<uint4 *>(P.codes) + m;
            const unsigned src0 = unsigned(P.bytes_at) + unsigned(ly * g.sh * P.bytes_pitch + lx * g.sw * g.C);
            const unsigned *words = reinterpret_cast<const unsigned *>(prep_smem);
            unsigned w[4] = {0, 0, 0, 0}, pending = 0;            // the last four words, and the bytes after them
            int count = 0, bits = 0;
            auto put = [&](unsigned v) {
                w[0] = w[1]; w[1] = w[2]; w[2] = w[3]; w[3] = v;
                if ((++count & 3) != 0) return;
                codes += int(__dp4a(w[0], 0x01010101u, __dp4a(w[1], 0x01010101u, __dp4a(w[2], 0x01010101u, __dp4a(w[3], 0x01010101u, 0u)))));
                if (AXC_SCRATCH_OK(P, dst, 16, 344u)) *dst = make_uint4(w[0] ^ zz, w[1] ^ zz, w[2] ^ zz, w[3] ^ zz);
                dst += g.M;
            };
            if (P.bytes_at < 0) {
                // a region that leaves no room for its codes: every tap's is computed again for each pixel that it belongs to
                for (int ky = 0; ky < g.KH; ++ky)
                    for (int kx = 0; kx < g.KW; ++kx) {
                        const float *src = prep_smem + (first + ky * g.dh * P.RW + kx * g.dw) * P.pitch;
                        if (!staged_ok(src - prep_smem, g.C, 346u)) continue;
                        for (int c = 0; c < g.C; ++c) {
                            pending |= code_of(src[c], q.in_off, q.in_inv) << bits;
                            if ((bits += 8) == 32) { put(pending); pending = 0; bits = 0; }
                        }
                    }
            } else
            for (int ky = 0; ky < g.KH; ++ky)
                for (int kx = 0; kx < runs_x; ++kx) {
                    const unsigned at = src0 + unsigned(ky * g.dh * P.bytes_pitch + kx * g.dw * g.C), shift = (at & 3u) * 8u;
                    if (!staged_ok(at >> 2, (run + 7) / 4, 339u)) continue;
                    const unsigned *src = words + (at >> 2);
                    unsigned lo = *src++;
                    for (int i = run >> 2; i > 0; --i) {
                        const unsigned hi = *src++, v = __funnelshift_r(lo, hi, shift);
                        lo = hi;
                        put(pending | v << bits);
                        pending = __funnelshift_rc(v, 0u, 32u - unsigned(bits));       // (a shift by 32 leaves nothing)
                    }
                    const int rest = (run & 3) * 8;
                    if (rest > 0) {
                        const unsigned v = __funnelshift_r(lo, *src, shift) & ((1u << rest) - 1u);
                        pending |= v << bits;
                        if ((bits += rest) >= 32) {
                            bits -= 32;
                            put(pending);
                            pending = __funnelshift_rc(v, 0u, unsigned(rest - bits));
                        }
                    }
                }
            if (bits > 0) put(pending);
            while (count & 3) put(0u);
        }
        if (P.sums && AXC_SCRATCH_OK(P, P.asum + m, 4, 340u)) P.asum[m] = s;
        if (P.acode && AXC_SCRATCH_OK(P, P.acode + m, 4, 341u)) P.acode[m] = codes;
    }
}

// ------------------------------------------------------------------------------------------------------------------
// expanded tables in global memory, for calls with enough pixels to use each of them several times
// ------------------------------------------------------------------------------------------------------------------
constexpr int kExpandThreads = 512;

struct ExpandParams {
    XGeom g;
    const float *filter;
    const uint8_t *filter_u8;
    const unsigned char *rows;      // table_rows_device: one row of entries per weight, row 256 all zeros
    const float *ranges;
    DevQuant host_q;
    unsigned char *xt;
    uint2 *wb;
    uint8_t *qf_debug;
    PlanHeader *hdr;
    long long scratch_bytes;
};

// xt[channel tile][chunk][row a][piece kk][16 bytes], kk = octet * 8 + k; 64 rows where they repeat, else 256.  The table's rows (one per weight) lie in shared memory.
// A lane reads the same word (two or four a) of the rows of its piece's 8 or 16 weights, transposes in registers and writes
// whole pieces; the 32 lanes (8 k x 4 words) read 32 different banks whatever the weights are, and write 128-byte runs.
// Bound by the writes, 64 KiB per chunk (gathering entry by entry with random banks took 12 700 clocks per chunk, this 1500); with 64 rows
// 16 KiB, so that two chunks share a turn of the CTA.
template <int MODE>
__global__ void __launch_bounds__(kExpandThreads, 1) xexpand_kernel(const ExpandParams P)
{
    constexpr int TNC = MODE == kXtabFull ? 8 : 16;
    constexpr unsigned kRow = MODE == kXtabFull ? 512u : MODE == kXtabByte ? 256u : 128u;     // bytes of a table row
    constexpr int kRounds = MODE == kXtabFull ? 64 : MODE == kXtabByte ? 32 : 8;               // warp rounds per chunk
    constexpr unsigned kRowsA = MODE == kXtabByte64 ? 64u : 256u;                              // rows of the expanded table
    extern __shared__ __align__(16) unsigned char expand_smem[];
    const XGeom &g = P.g;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned tab = (unsigned)__cvta_generic_to_shared(expand_smem), lists = tab + 257u * kRow, bar = lists + (MODE == kXtabByte64 ? 4u : 2u) * 16u * TNC * 2u;
    pdl_trigger();
    if (tid == 0) {
        mbar_init(bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(257u * kRow) : "memory");
        bulk_copy(tab, P.rows, 257u * kRow, bar);
    }
    __syncthreads();
    const DevQuant q = P.ranges ? dev_quant_from_ranges(P.ranges, g.K) : P.host_q;
    const unsigned z = code_of(0.0f, q.in_off, q.in_inv) & (kRowsA - 1u);
    bool ok = true;
    mbar_wait(bar, 0u, ok, AXC_WAIT_POLLS(0));
    // thread (kk, slot) of the first 16*TNC prepares the list of table rows of a chunk
    const int kk = tid / TNC % 16, slot = tid % TNC;
    const int elem = ((kk & 3) << 2) + ((kk >> 3) << 1) + ((kk >> 2) & 1);           // element 4t + 2*octet + p
    const int total = g.tiles_n * g.chunks;
    const int kidx = lane & 7, sub = lane >> 3;
    unsigned parity = 0;
    constexpr int kTurn = MODE == kXtabByte64 ? 2 : 1;             // chunks at a time (256 rows: one occupies all warps)
    const unsigned my_lists = lists + unsigned(tid / (16 * TNC)) * (16u * TNC * 2u);
    for (int tc0 = int(blockIdx.x) * kTurn; tc0 < total; tc0 += int(gridDim.x) * kTurn, parity ^= 1u) {
        const int tc = tc0 + tid / (16 * TNC);
        if (tid < 16 * TNC * kTurn && tc < total) {
            const int nt = tc / g.chunks, ch = tc - nt * g.chunks;
            const int k = k_of(g, ch, elem), cj = slot_channel(MODE, slot), j = nt * TNC + cj;
            unsigned row = kNull;
            if (k >= 0 && j < g.Cout) {
                row = code_of(P.filter_u8 ? filter_value<true>(g, P.filter, P.filter_u8, (size_t)k * g.Cout + j) : filter_value<false>(g, P.filter, P.filter_u8, (size_t)k * g.Cout + j), q.f_off, q.f_inv);
                if (P.qf_debug) P.qf_debug[(size_t)k * g.Cout + j] = uint8_t(row);
            }
            if (AXC_SHARED_OK(my_lists + parity * (16u * TNC * 2u * kTurn) + unsigned(kk * TNC + slot) * 2u, 2u, lists, bar, 350u))
                asm volatile("st.shared.u16 [%0], %1;" ::"r"(my_lists + parity * (16u * TNC * 2u * kTurn) + unsigned(kk * TNC + slot) * 2u), "h"((unsigned short)row) : "memory");
            if (MODE != kXtabFull) {
                // exact products, B operand half h, column n: channel (n>>1)*4 + 2h + (n&1); lane (n, t) holds elements 4t..4t+3
                const int t = elem >> 2, h = (cj >> 1) & 1, n = (cj >> 2) * 2 + (cj & 1);
                unsigned char *w = reinterpret_cast<unsigned char *>(P.wb + (size_t)tc * 32 + n * 4 + t) + h * 4 + (elem & 3);
                if (AXC_SCRATCH_OK(P, w, 1, 351u)) *w = row == kNull ? 0 : (unsigned char)row;
            }
        }
        __syncthreads();                                           // (the other list's readers are a chunk behind this barrier)
        for (int r0 = warp; r0 < kRounds * kTurn; r0 += kExpandThreads / 32) {
            const int r = r0 % kRounds, o = r / (kRounds / 2), x = r % (kRounds / 2);     // octet, round
            const int tc = tc0 + r0 / kRounds;
            if (tc >= total) continue;
            const unsigned word = unsigned((x >> 3) * 32 + ((4 * ((x & 7) + kidx) + sub) & 31));
            const unsigned list = lists + (parity * kTurn + unsigned(r0 / kRounds)) * (16u * TNC * 2u) + unsigned((o * 8 + kidx) * TNC) * 2u;
            unsigned v[TNC];
#pragma unroll
            for (int s4 = 0; s4 < TNC / 8; ++s4) {
                const uint4 l = lds128(list + unsigned(s4) * 16u);
                const unsigned l4[4] = {l.x, l.y, l.z, l.w};
#pragma unroll
                for (int s = 0; s < 8; ++s) v[s4 * 8 + s] = lds32(tab + ((s & 1) ? l4[s >> 1] >> 16 : l4[s >> 1] & 0xFFFFu) * kRow + word * 4u);
            }
            uint4 *dst = reinterpret_cast<uint4 *>(P.xt + (size_t)tc * (kRowsA * 256u)) + o * 8 + kidx;
            if (!AXC_SCRATCH_OK(P, dst, (kRowsA - 1u) * 256 + 16, 352u)) continue;      // the rows a of this piece
            if (MODE == kXtabFull) {
                const unsigned a = word * 2u;
                dst[(a ^ z) * 16u] = make_uint4(prmt<0x5410>(v[0], v[1]), prmt<0x5410>(v[2], v[3]), prmt<0x5410>(v[4], v[5]), prmt<0x5410>(v[6], v[7]));
                dst[((a + 1u) ^ z) * 16u] = make_uint4(prmt<0x7632>(v[0], v[1]), prmt<0x7632>(v[2], v[3]), prmt<0x7632>(v[4], v[5]), prmt<0x7632>(v[6], v[7]));
            } else {
                unsigned w4[4][4];                                 // [row a][word]
#pragma unroll
                for (int w = 0; w < TNC / 4; ++w) {
                    const unsigned t0 = prmt<0x5140>(v[4 * w], v[4 * w + 1]), t1 = prmt<0x5140>(v[4 * w + 2], v[4 * w + 3]);
                    const unsigned t2 = prmt<0x7362>(v[4 * w], v[4 * w + 1]), t3 = prmt<0x7362>(v[4 * w + 2], v[4 * w + 3]);
                    w4[0][w] = prmt<0x5410>(t0, t1); w4[1][w] = prmt<0x7632>(t0, t1);
                    w4[2][w] = prmt<0x5410>(t2, t3); w4[3][w] = prmt<0x7632>(t2, t3);
                }
#pragma unroll
                for (unsigned i = 0; i < 4; ++i) dst[(((word * 4u + i) & (kRowsA - 1u)) ^ z) * 16u] = make_uint4(w4[i][0], w4[i][1], w4[i][2], w4[i][TNC / 4 - 1]);
            }
        }
    }
    pdl_wait();                                                    // the kernel after this one waits for this one only
    if (!ok) {
        if (tid == 0) mbar_drain(bar, 0u);
        atomicExch(&P.hdr->status, 3);                             // (xprep_kernel, which clears it, is complete)
    }
}

// ------------------------------------------------------------------------------------------------------------------
// the convolution
// ------------------------------------------------------------------------------------------------------------------
struct XParams {
    XGeom g;
    const unsigned char *codes, *tt;
    const uint16_t *wrow;
    const uint2 *wb;
    const unsigned char *xt;    // expanded tables [channel tile][chunk][256 or 64 rows][2 octets][8][16], or NULL: built by the CTAs
    const float *asum, *bsum;
    const PlanHeader *hdr;
    long long scratch_bytes;
    float *output;              // NULL: integer sums only
    int32_t *acc_out;
    int32_t *partial;           // K split over CTAs: integer sums are added here
    const float *bias, *residual;
    float out_floor;
    int plain;                  // one output (fp32 or the integer sums), it and the shortcut at 16-byte boundaries
    int k_e_min;                // K times what every entry was stored less
    const int *acode, *bcode;   // sums of codes (or NULL) and what they enter the total with: 128 for a centred table, less
    int a_coef, b_coef;         // the zero points of a quantised call
    int splits, chunks_per_split;
    int group;                  // units that a CTA takes one after the other: neighbouring pixels, the same channels and part of K
    long long units;            // pixel tiles x channel tiles x splits
};

// ((S*s1s2 + m2*aSum) + m1*bSum) - K*m1m2, then what the op's callers add
__device__ __forceinline__ float dequantise(const DevQuant &Q, int total, float a_sum, float t2)
{
    return __fsub_rn(__fadd_rn(__fadd_rn(__fmul_rn(float(total), Q.s1s2), __fmul_rn(Q.m2, a_sum)), t2), Q.km1m2);
}

// MODE: XtabMode.  NB: blocks of 8 pixels per warp (tile = 64*NB pixels).
// Warp w holds the sums of pixels [w*8*NB, (w+1)*8*NB) x all channels of the tile in 2*NB (16-bit entries) or 4*NB registers
// per lane.  Lane (g, t) = (lane / 4, lane % 4) looks pixel g of a block up at k = t and t + 4 of an octet; even and odd g take
// the two in opposite order, so that a quarter warp covers all 8 k at once.
// All warps are alike: each builds an eighth of the next octet's expanded table, in four rounds between its own lookups (64 rows: four
// warps, a quarter each in two rounds), and fetches the codes of its own pixels.  Eight warps with 255 registers rather than sixteen with 128: the loads of the next two
// block pairs are in flight while the MMAs of the last two run.
// PRE: the expanded tables come from global memory (xexpand_kernel) by bulk copies, 64 KiB per 16 elements of K, which cost the
// shared-memory pipe next to nothing (measured: 2 to 4 % beside a stream of LDS.128 + MMA); otherwise they are built here.
// W: warps.  Where the rows repeat, an expanded table is a quarter as large and half of a tile and its tables fit half of an SM: two
// CTAs of four warps then, and one looks up while the other waits, starts or ends a tile.
template <int MODE>
constexpr int kWarpsOf = MODE == kXtabByte64 ? 4 : kWarps;

template <int MODE, int NB, bool PRE>
__global__ void __launch_bounds__(kWarpsOf<MODE> * 32, MODE == kXtabByte64 ? 2 : 1) xtab_kernel(const XParams P)
{
    constexpr int W = kWarpsOf<MODE>;
    constexpr int kPix = W * 8 * NB;
    constexpr int TNC = MODE == kXtabFull ? 8 : 16, HV = TNC / 8;
    constexpr bool kTables = MODE != kXtabExact, kBuild = kTables && !PRE;
    constexpr bool kSmall = MODE == kXtabByte64, kBytes = kSmall || MODE == kXtabByte;
    constexpr unsigned kChunkTable = kSmall ? 16384u : 65536u;     // expanded table of 16 elements of K
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const XGeom &g = P.g;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned dyn0 = (unsigned)__cvta_generic_to_shared(smem_raw);
    unsigned dyn_size;
    asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dyn_size));
    const unsigned bars = (dyn0 + 15u) & ~15u;
    const unsigned tab_full = bars, tab_empty = bars + 32u, rows_full = bars + 64u, asked = bars + 72u;
    pdl_trigger();
    pdl_wait();
    if (asked + 4u > kCodes || dyn0 + dyn_size < (kSmall ? kWindowHalf : kWindowEnd)) {
        if (tid == 0) atomicExch(const_cast<int *>(&P.hdr->status), 2);      // (xprep_kernel, which clears it, is complete)
        return;
    }
    if (tid == 0) {
        if (PRE) asm volatile("st.shared.u32 [%0], %1;" ::"r"(asked), "r"(0xFFFFFFFFu) : "memory");
        for (int s = 0; s < 2; ++s) { mbar_init(tab_full + s * 8, PRE ? 1 : W); mbar_init(tab_empty + s * 8, W); }
        mbar_init(rows_full, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        if (kBuild) {
            // the transposed table stays for the CTA's lifetime
            constexpr unsigned low = MODE == kXtabFull ? kLowRows * 512u : 0u, high = MODE == kXtabFull ? (257u - kLowRows) * 512u : 257u * (kSmall ? 128u : 256u);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(rows_full), "r"(low + high) : "memory");
            if (low > 0) bulk_copy(kRowsLow, P.tt, low, rows_full);
            bulk_copy(kSmall ? kRowsSmall : kRowsHigh, P.tt + low, high, rows_full);
        }
    }
    __syncthreads();
    bool ok = true;
    const unsigned units = unsigned(P.units);

    // unit number -> split of K, channel tile, first pixel, chunks
    auto coords = [&](unsigned u, int &nt, int &m0, int &c_begin, int &c_end) {
        const unsigned v = kSmall ? u / unsigned(P.group) : u, sub = kSmall ? u - v * unsigned(P.group) : 0u;
        const unsigned u2 = v / unsigned(P.splits), sp = v - u2 * unsigned(P.splits), mt = u2 / unsigned(g.tiles_n);
        nt = int(u2 - mt * unsigned(g.tiles_n));
        m0 = int(kSmall ? mt * unsigned(P.group) + sub : mt) * kPix;
        c_begin = int(sp) * P.chunks_per_split;
        c_end = min(g.chunks, c_begin + P.chunks_per_split);
    };

    const unsigned first_unit = kSmall ? blockIdx.x * unsigned(P.group) : blockIdx.x;
    auto after = [&](unsigned u) {                                 // the unit that this CTA takes after unit u
        if (!kSmall) return u + gridDim.x;
        return (u + 1u) % unsigned(P.group) != 0u ? u + 1u : u + 1u + (gridDim.x - 1u) * unsigned(P.group);
    };

    // ---- codes: this warp's pixels, 16 elements of K at a time ---------------------------------------------------------
    // Asked for kAhead chunks before they are used: a chunk of a small tile is over before memory has answered.
    constexpr int kAhead = !kTables ? 1 : NB <= 8 ? 4 : NB == 16 ? 2 : 1;
    unsigned chunk = 0;                                            // chunks of this CTA so far
    constexpr int PPL = (NB * 8 + 31) / 32;                        // pixels per lane
    const int pieces = g.im2col ? g.M : g.N * g.H * g.W;           // distance of the 16-byte pieces of one pixel
    const int eh = g.im2col ? 1 : g.H, ew = g.im2col ? 1 : g.W;
    const unsigned my_codes = kCodes + unsigned(warp) * (NB * 8 * 16u);
    int f_base[PPL], f_yx[PPL];                                    // pixel number of the patch origin, its row and column
    unsigned f_unit = first_unit;
    int f_left = 0, f_cc = 0, f_ky = 0, f_kx = 0;
    auto fetch_unit = [&]() {
        int nt, m0, c_begin, c_end;
        coords(f_unit, nt, m0, c_begin, c_end);
        f_left = c_end - c_begin;
        f_cc = c_begin; f_ky = 0; f_kx = 0;
        if (!g.im2col) {
            const int tap = c_begin / g.CC;
            f_cc = c_begin - tap * g.CC;
            f_ky = tap / g.KW;
            f_kx = tap - f_ky * g.KW;
        }
#pragma unroll
        for (int i = 0; i < PPL; ++i) {
            const int m = m0 + warp * (NB * 8) + i * 32 + lane;
            int b = 0, y = -32768, x = 0;                          // no pixel: every tap out of range
            if (m < g.M && i * 32 + lane < NB * 8) {
                b = m; y = 0;
                if (!g.im2col) {
                    const unsigned mm = unsigned(m), row = mm / unsigned(g.OW), n = row / unsigned(g.OH);
                    y = int(row - n * unsigned(g.OH)) * g.sh - g.ph;
                    x = int(mm - row * unsigned(g.OW)) * g.sw - g.pw;
                    b = (int(n) * g.H + y) * g.W + x;
                }
            }
            f_base[i] = b;
            f_yx[i] = (y << 16) | (x & 0xFFFF);
        }
    };
    // One chunk is asked for in PPL pieces (the caller spreads them over its lookups): fetch_begin() finds the chunk,
    // fetch_pixel(i, dst) asks for the lane's i-th pixel.
    bool f_active = false;
    int f_off = 0, f_dy = 0, f_dx = 0;
    auto fetch_begin = [&]() {
        f_active = false;
        if (f_left == 0) {
            f_unit = after(f_unit);
            if (f_unit >= units) return;
            fetch_unit();
        }
        f_active = true;
        f_dy = f_ky * g.dh; f_dx = f_kx * g.dw;
        f_off = f_dy * g.W + f_dx + f_cc * pieces;
        if (++f_cc == g.CC && !g.im2col) { f_cc = 0; if (++f_kx == g.KW) { f_kx = 0; ++f_ky; } }
        --f_left;
    };
    auto fetch_pixel = [&](int i, unsigned dst) {
        if (!f_active || (NB * 8 < 32 && lane >= NB * 8)) return;
        const bool in = unsigned((f_yx[i] >> 16) + f_dy) < unsigned(eh) && unsigned(int(short(f_yx[i])) + f_dx) < unsigned(ew) &&
                        AXC_GLOBAL_OK(f_base[i] + f_off, (long long)pieces * g.CC, 310u);
        cp_async16(dst + unsigned(i * 32 + lane) * 16u, P.codes + (in ? (size_t)unsigned(f_base[i] + f_off) * 16u : 0u), in ? 16u : 0u);
    };
    auto fetch_chunk = [&](unsigned dst) {
        fetch_begin();
#pragma unroll
        for (int i = 0; i < PPL; ++i) fetch_pixel(i, dst);
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    // ---- expanded tables: this warp's eighth, one octet ahead ----------------------------------------------------------
    // Round r: a lane reads one word of the rows of 8 weights of element kidx (two a of 16-bit entries, four a of 8-bit
    // entries, whose 16 channels are shared by two lanes) and writes the expanded rows of those a.  The 32 lanes read 32
    // different banks, whatever the weights, and write different bank groups.
    const int kidx = lane & 7, sub = lane >> 3;
    const int hf = kBytes ? sub & 1 : 0;
    unsigned raw[8];
    unsigned b_unit = first_unit;
    int b_left = 0;                                                // octets left to build in b_unit
    const uint4 *b_rows = nullptr;
    constexpr int kLists = NB < 32 ? 2 : 1;                        // row lists asked for ahead (the largest tiles have no registers to spare)
    uint4 wq = make_uint4(0, 0, 0, 0), wq_next[2] = {wq, wq};      // of the octet being built and of those after it
    auto build_unit = [&]() {
        int nt, m0, c_begin, c_end;
        coords(b_unit, nt, m0, c_begin, c_end);
        b_left = 2 * (c_end - c_begin);
        b_rows = reinterpret_cast<const uint4 *>(P.wrow) + (((size_t)nt * g.chunks + c_begin) * 16 + kidx) * HV + hf;
    };
    auto build_ask = [&](int h) {                                  // request the next octet's row list (octet h of a chunk)
        if (b_left == 0) {
            b_unit = after(b_unit);
            if (b_unit >= units) return;
            build_unit();
        }
        if (AXC_SCRATCH_OK(P, b_rows, 16, 312u)) wq_next[h & (kLists - 1)] = __ldg(b_rows);
        b_rows += 8 * HV;
        --b_left;
    };
    auto build_next = [&](int h) {                                 // take an octet's row list, request the next one that has not been
        wq = wq_next[h & (kLists - 1)];
        build_ask(h);
    };
    // Words of a row that the lane works on: 32 r + (4 (warp + kidx) + sub) mod 32 in round r (8-bit entries: 32 (r / 2) + .. with
    // the two lanes that share a piece's channels swapped in odd rounds), so that a round is a constant offset.
    // Rows that repeat have 16 words, kept twice: two rounds of the four warps cover them, the lanes of the second copy with the low
    // bit swapped so that both channel halves meet all of them.
    const unsigned turn = (unsigned(warp) + unsigned(kidx)) & 7u;
    const unsigned word0 = 4u * turn + (kSmall ? unsigned(sub) ^ (turn >> 2) : unsigned(sub)), word1 = word0 ^ 1u;
    unsigned row_at[8];
    auto build_rows = [&]() {
        const unsigned w4[4] = {wq.x, wq.y, wq.z, wq.w};
#pragma unroll
        for (int s = 0; s < 8; ++s) row_at[s] = ((s & 1) ? w4[s >> 1] >> 16 : w4[s >> 1] & 0xFFFFu) * 16u + word0 * 4u;
    };
    auto build_load = [&](int r) {
        const unsigned odd = kSmall && r == 1 ? (word0 ^ 17u) * 4u - word0 * 4u : kBytes && (r & 1) ? word1 * 4u - word0 * 4u : 0u;
#pragma unroll
        for (int s = 0; s < 8; ++s) raw[s] = lds32(row_at[s] + odd + (kBytes ? unsigned(r >> 1) : unsigned(r)) * 128u);
    };
    auto build_store = [&](int r, unsigned st) {
        // (rows that repeat: st = the octet's place among the 4 of two chunks, two to a row of 256 bytes)
        const unsigned word = kSmall ? (word0 ^ unsigned(r)) & 15u : kBytes && (r & 1) ? word1 : word0;
        const unsigned dst = kTab + (kSmall ? (st >> 1) * kChunkTable + (st & 1u) * 128u : st * 128u) + unsigned(kidx) * 16u + unsigned(hf) * 8u +
                             (MODE == kXtabFull ? word * 512u + unsigned(r) * 16384u : word * 1024u + (kSmall ? 0u : unsigned(r >> 1) * 32768u));
        if (MODE == kXtabFull) {
            sts128(dst, make_uint4(prmt<0x5410>(raw[0], raw[1]), prmt<0x5410>(raw[2], raw[3]), prmt<0x5410>(raw[4], raw[5]), prmt<0x5410>(raw[6], raw[7])));
            sts128(dst + 256u, make_uint4(prmt<0x7632>(raw[0], raw[1]), prmt<0x7632>(raw[2], raw[3]), prmt<0x7632>(raw[4], raw[5]), prmt<0x7632>(raw[6], raw[7])));
        } else {
            unsigned o[4][2];                                      // [row a][word]
#pragma unroll
            for (int w = 0; w < 2; ++w) {
                const unsigned t0 = prmt<0x5140>(raw[4 * w], raw[4 * w + 1]), t1 = prmt<0x5140>(raw[4 * w + 2], raw[4 * w + 3]);
                const unsigned t2 = prmt<0x7362>(raw[4 * w], raw[4 * w + 1]), t3 = prmt<0x7362>(raw[4 * w + 2], raw[4 * w + 3]);
                o[0][w] = prmt<0x5410>(t0, t1); o[1][w] = prmt<0x7632>(t0, t1);
                o[2][w] = prmt<0x5410>(t2, t3); o[3][w] = prmt<0x7632>(t2, t3);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) sts64(dst + unsigned(i) * 256u, o[i][0], o[i][1]);
        }
    };

    // ---- expanded tables from global memory: two chunks in flight, issued by one thread ------------------------------------
    unsigned x_unit = first_unit;
    int x_left = 0;
    const unsigned char *x_src = nullptr;
    auto copy_table = [&](unsigned buf) {                          // the next chunk's table into buffer `buf`
        if (x_left == 0) {
            if (x_src) x_unit = after(x_unit);
            if (x_unit >= units) return;
            int nt, m0, c_begin, c_end;
            coords(x_unit, nt, m0, c_begin, c_end);
            x_left = c_end - c_begin;
            x_src = P.xt + ((size_t)nt * g.chunks + c_begin) * kChunkTable;
        }
        if (!AXC_SCRATCH_OK(P, x_src, kChunkTable, 311u)) { ok = false; return; }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(tab_full + buf * 8), "r"(kChunkTable) : "memory");
        bulk_copy(kSmall ? kTab + buf * kChunkTable : kTab * (1u + buf), x_src, kChunkTable, tab_full + buf * 8);
        x_src += kChunkTable;
        --x_left;
    };

    // ---- lookups ---------------------------------------------------------------------------------------------------------
    const int gr = lane >> 2, t = lane & 3;
    const DevQuant Q = *reinterpret_cast<const DevQuant *>(reinterpret_cast<const unsigned char *>(P.hdr) + kDevQuantOffset);
    const unsigned zz = code_of(0.0f, Q.in_off, Q.in_inv) * 0x01010101u;
    // Constant B operands.  A row of A has the words x, z of a piece, the row eight below it y, w.  8-bit entries: column n
    // adds byte n of (x, z) resp. (y, w): 16 channels.  16-bit entries: digits 1 and 255 of the two channels of a word,
    // in columns 0..3 for the first block of a pair, 4..7 for the second: one accumulator fragment serves both.
    unsigned b00, b01, b10, b11;
    if (MODE == kXtabFull) {
        const unsigned digits = (gr & 1) ? 0xFF010000u : 0x0000FF01u;
        b00 = (gr >> 1) == 0 ? digits : 0u; b01 = (gr >> 1) == 1 ? digits : 0u;
        b10 = (gr >> 1) == 2 ? digits : 0u; b11 = (gr >> 1) == 3 ? digits : 0u;
    } else {
        b00 = b10 = gr < 4 ? 1u << (8 * gr) : 0u;
        b01 = b11 = gr >= 4 ? 1u << (8 * (gr - 4)) : 0u;
    }
    // step s of an octet: even pixels take k = t + 4s, odd ones t + 4(1 - s)
    const unsigned p0 = unsigned(gr & 1);
    const unsigned lane_k0 = kTab + unsigned(t + 4 * p0) * 16u, lane_k1 = kTab + unsigned(t + 4 * (1 - p0)) * 16u;
    constexpr int kAcc = NB * HV / 2;                              // accumulator fragments
    int acc[kAcc][4];
    unsigned cw[NB];
    // Octet h (0 / 1) of the chunk, from the table of stage st; `more`: build the next octet's table into the other stage.
    // Steps of two block pairs and one of their two k: the loads of a step are issued before the MMAs of the step before it,
    // and no MMA waits for the one just issued (16-bit entries: two MMAs per pair and step add into one accumulator).
    // Spread over the steps as well, so that the shared-memory pipe never waits for them (measured as bursts at the chunk's
    // start: 830 clocks per octet of 2048 pixels): one MMA of the exact products per step; in octet 0 the requests for the next
    // chunk's codes; in octet 1, where the last use of a code has passed, the loads of the next chunk's; four rounds of building.
    constexpr int kSteps = NB / 2;
    const unsigned code_src = my_codes + unsigned(gr) * 16u + unsigned(t) * 4u;
    auto product = [&](int i, uint2 wb) {                          // both rows of a pixel hold its codes, each against half of the channels
        const unsigned q = cw[i] ^ zz;
        mma_k32(acc[i * HV / 2], q, 0u, 0u, q, wb.x, wb.y);
    };
    unsigned ring = 0;                                             // rows that repeat: place of the chunk's table, in the upper bits of every code byte
    auto row_of = [&](unsigned codes) { return kSmall ? (codes & 0x3F3F3F3Fu) | ring : codes; };
    auto octet = [&](int h, unsigned toff, unsigned st, unsigned oct, bool more, uint2 wb) {
        const unsigned l0 = lane_k0 + toff, l1 = lane_k1 + toff;
        // address = {low byte of l, code byte, upper half of l}
        const unsigned s0 = 0x3200u | ((4u + 2u * h + p0) << 4), s1 = 0x3200u | ((4u + 2u * h + 1u - p0) << 4);
        uint4 x[2][4];
        auto request = [&](int n, uint4 (&v)[4]) {
            const int i = (n >> 1) * 2;                            // pairs i, i + 1
#pragma unroll
            for (int e = 0; e < 4; ++e) v[e] = lds128((n & 1) ? prmt_r(l1, row_of(cw[2 * i + e]), s1) : prmt_r(l0, row_of(cw[2 * i + e]), s0));
        };
        request(0, x[0]);
        if (h == 0) fetch_begin();
        else {
            if (kAhead > 1) asm volatile("cp.async.wait_group %0;" ::"n"(kAhead - 1) : "memory");
            else asm volatile("cp.async.wait_all;" ::: "memory");
            __syncwarp();
        }
#pragma unroll
        for (int n = 0; n < kSteps; ++n) {
            if (n + 1 < kSteps) request(n + 1, x[(n + 1) & 1]);
            const int i = (n >> 1) * 2;
            uint4 (&v)[4] = x[n & 1];
            // a loaded piece is an A operand as it is
            mma_k32(acc[i * HV], v[0].x, v[0].y, v[0].z, v[0].w, b00, b01);
            mma_k32(acc[(i + 1) * HV], v[2].x, v[2].y, v[2].z, v[2].w, b00, b01);
            mma_k32(acc[i * HV + HV - 1], v[1].x, v[1].y, v[1].z, v[1].w, b10, b11);
            mma_k32(acc[(i + 1) * HV + HV - 1], v[3].x, v[3].y, v[3].z, v[3].w, b10, b11);
            if (MODE != kXtabFull) product(h * kSteps + n, wb);
            if (h == 0) {
#pragma unroll
                for (int f = 0; f < PPL; ++f)
                    if (n == f * kSteps / PPL) fetch_pixel(f, kAhead > 1 ? my_codes + (chunk & (kAhead - 1)) * (kPix * 16u) : my_codes);
            } else if (n & 1) {
#pragma unroll
                for (int e = 0; e < 4; ++e) cw[2 * (n - 1) + e] = lds32((kAhead > 1 ? code_src + ((chunk + 1u) & (kAhead - 1)) * (kPix * 16u) : code_src) + unsigned(2 * (n - 1) + e) * 128u);
            }
            if (PRE && h == 0 && n == 1 && tid == 0 && oct > 0) {
                // the other buffer's readers finished the chunk before this one: ask for the chunk after this one
                mbar_wait(tab_empty + (st ^ 1u) * 8, ((oct - 1) >> 1) & 1u, ok, AXC_WAIT_POLLS(1));
                if (ok) copy_table(st ^ 1u);
                else asm volatile("st.shared.u32 [%0], %1;" ::"r"(asked), "r"(min(lds32(asked), oct + 1u)) : "memory");   // the buffer's last copy may be in flight
            }
            if (kBuild && kSmall && more) {                            // oct: chunk; octet h of the next one, in two rounds
                if (n == 0) {
                    build_next(h);
                    // the place's last readers worked on the chunk before this one
                    if (h == 0 && oct > 0) mbar_wait(tab_empty + ((oct + 1u) & 1u) * 8, ((oct - 1u) >> 1) & 1u, ok, AXC_WAIT_POLLS(1));
                    build_rows();
                    build_load(0);
                }
                if (n == (kSteps < 4 ? 1 : 2)) {
                    build_store(0, ((oct + 1u) & 1u) * 2u + unsigned(h));
                    build_load(1);
                }
                if (n == kSteps - 1) build_store(1, ((oct + 1u) & 1u) * 2u + unsigned(h));
            } else if (kBuild && more) {
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    if (n == r * kSteps / 4) {
                        if (r == 0) {
                            build_next(h ^ 1);
                            // the stage's last readers worked on the octet before this one
                            if (oct > 0) mbar_wait(tab_empty + (st ^ 1u) * 8, ((oct - 1) >> 1) & 1u, ok, AXC_WAIT_POLLS(1));
                            build_rows();
                        }
                        build_load(r);
                    }
                    if (n == (kSteps < 4 ? r * kSteps / 4 : (r + 1) * kSteps / 4 - 1)) build_store(r, st ^ 1u);
                }
            }
        }
        if (kAhead > 1 && h == 0) asm volatile("cp.async.commit_group;" ::: "memory");
        __syncwarp();                                              // also: every lane has the codes before the next are asked for
        if (lane == 0) {
            if (kBuild && kSmall) {
                if (h == 1 && more) mbar_arrive(tab_full + ((oct + 1u) & 1u) * 8);
                if (h == 1) mbar_arrive(tab_empty + (oct & 1u) * 8);
            } else {
                if (kBuild && more) mbar_arrive(tab_full + (st ^ 1u) * 8);
                if (kBuild || h == 1) mbar_arrive(tab_empty + st * 8);
            }
        }
    };

    unsigned oct = 0, oct_total = 0;                               // octets of this CTA so far, and all of them
    constexpr int kBufs = kTables ? 1 : 4;                         // code buffers (only exact products: latency is all there is)
    if (first_unit < units) {
        fetch_unit();
#pragma unroll
        for (int k = 0; k < (kTables ? kAhead : kBufs - 1); ++k) fetch_chunk(my_codes + unsigned(k) * (kPix * 16u));
    }
    if (kTables && first_unit < units) {
        for (unsigned u = first_unit; u < units; u = after(u)) {
            int nt, m0, c_begin, c_end;
            coords(u, nt, m0, c_begin, c_end);
            oct_total += 2u * unsigned(c_end - c_begin);
        }
        if (PRE && tid == 0) {
            copy_table(0u);
            copy_table(1u);
        }
        if (kBuild) {
            build_unit();
            build_ask(0);
            if (kLists > 1) build_ask(1);
            mbar_wait(rows_full, 0u, ok, AXC_WAIT_POLLS(1));
            if (kSmall) {
#pragma unroll
                for (unsigned o = 0; o < 2u; ++o) {                       // a chunk
                    build_next(int(o));
                    build_rows();
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        build_load(r);
                        build_store(r, o);
                    }
                }
            } else {
                build_next(0);
                build_rows();
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    build_load(r);
                    build_store(r, 0u);
                }
            }
        }
        asm volatile("cp.async.wait_group %0;" ::"n"(kAhead - 1) : "memory");
        __syncwarp();
        if (kBuild && lane == 0) mbar_arrive(tab_full);
#pragma unroll
        for (int i = 0; i < NB; ++i) cw[i] = lds32(code_src + unsigned(i) * 128u);
        __syncwarp();
    }
    for (unsigned u = first_unit; u < units; u = after(u)) {
        int nt, m0, c_begin, c_end;
        coords(u, nt, m0, c_begin, c_end);
#pragma unroll
        for (int i = 0; i < kAcc; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[i][e] = 0;
        // the shortcut is read at the tile's end, four loads at a time: from L2 by then (not in the form that spills registers as it is)
        if (!(MODE == kXtabByte && NB == 32 && kBuild) && P.residual && !P.partial) {
#pragma unroll 1
            for (int p = warp * (NB * 8) + lane; p < (warp + 1) * (NB * 8) && m0 + p < g.M; p += 32)
                asm volatile("prefetch.global.L2 [%0];" ::"l"(P.residual + (size_t)(m0 + p) * g.Cout + nt * TNC));
        }
        const uint2 *wbp = P.wb + ((size_t)nt * g.chunks + c_begin) * 32 + lane;
        uint2 wb_next = make_uint2(0, 0);
        if (MODE != kXtabFull && AXC_SCRATCH_OK(P, wbp, 8, 316u)) wb_next = __ldg(wbp);
        for (int c = c_begin; c < c_end; ++c, ++chunk) {
            const uint2 wb = wb_next;
            wbp += 32;
            if (MODE != kXtabFull && c + 1 < c_end && AXC_SCRATCH_OK(P, wbp, 8, 317u)) wb_next = __ldg(wbp);
            if (PRE) {
                const unsigned st = chunk & 1u;
                ring = st * 0x40404040u;
                mbar_wait(tab_full + st * 8, (chunk >> 1) & 1u, ok, AXC_WAIT_POLLS(1));
#pragma unroll
                for (int h = 0; h < 2; ++h) octet(h, (kSmall ? 0u : st * kTab) + unsigned(h) * 128u, st, chunk, true, wb);
            } else if (kTables && kSmall) {
                ring = (chunk & 1u) * 0x40404040u;
                mbar_wait(tab_full + (chunk & 1u) * 8, (chunk >> 1) & 1u, ok, AXC_WAIT_POLLS(1));
#pragma unroll
                for (int h = 0; h < 2; ++h) octet(h, unsigned(h) * 128u, 0u, chunk, 2u * chunk + 2u < oct_total, wb);
            } else if (kTables) {
#pragma unroll
                for (int h = 0; h < 2; ++h, ++oct) {
                    mbar_wait(tab_full + (oct & 1u) * 8, (oct >> 1) & 1u, ok, AXC_WAIT_POLLS(1));
                    octet(h, (oct & 1u) * 128u, oct & 1u, oct, oct + 1 < oct_total, wb);
                }
            } else {
                asm volatile("cp.async.wait_group %0;" ::"n"(kBufs - 2) : "memory");
                __syncwarp();
                const unsigned src = code_src + (chunk & (kBufs - 1)) * (kPix * 16u);
#pragma unroll
                for (int i = 0; i < NB; ++i) cw[i] = lds32(src + unsigned(i) * 128u);
                __syncwarp();
                fetch_chunk(my_codes + ((chunk + kBufs - 1) & (kBufs - 1)) * (kPix * 16u));
#pragma unroll
                for (int i = 0; i < NB; ++i) product(i, wb);
            }
        }
        // ---- dequantise and store: a fragment is four neighbouring channels of one pixel -------------------------------
        const int j0 = nt * TNC + 4 * (MODE == kXtabFull ? t & 1 : t);
        float t2[4], bias[4];
        int back[4];                                               // what the stored entries lack: per channel
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            t2[e] = (!P.partial && j0 + e < g.Cout) ? __fmul_rn(Q.m1, __ldg(P.bsum + j0 + e)) : 0.0f;
            bias[e] = (P.bias && j0 + e < g.Cout) ? __ldg(P.bias + j0 + e) : 0.0f;
            back[e] = P.k_e_min + (P.bcode && j0 + e < g.Cout ? P.b_coef * __ldg(P.bcode + j0 + e) : 0);
        }
        const bool whole = j0 + 4 <= g.Cout && (g.Cout & 3) == 0, chan = j0 < g.Cout;
        constexpr int EB = kAcc < 4 ? kAcc : 4;
        constexpr int kStep = MODE == kXtabFull ? 16 : 8;          // pixels from fragment to fragment
        const int first = warp * (NB * 8) + gr + (MODE == kXtabFull ? (t >> 1) * 8 : 0);
        int left = chan ? g.M - m0 - first : 0;                    // > kStep * i: fragment i has a pixel
        if (left > 0 && !P.partial && !AXC_SCRATCH_OK(P, P.asum + g.M - 1, 4, 318u)) left = 0;
        if (left > 0 && P.acode && !AXC_SCRATCH_OK(P, P.acode + g.M - 1, 4, 319u)) left = 0;
        const long long at0 = (long long)(m0 + first) * g.Cout + j0;
        const int row = kStep * g.Cout;
        if (P.partial && whole) {
            // K split over CTAs: nothing but the additions, in as few instructions as the other cases below
            int32_t *sums = P.partial + at0;
#pragma unroll
            for (int i = 0; i < kAcc; ++i) {
                if (i * kStep >= left || !AXC_SCRATCH_OK(P, sums + i * row, 16, 342u)) continue;
#pragma unroll
                for (int e = 0; e < 4; ++e) atomicAdd(sums + i * row + e, acc[i][e]);
            }
        } else if (P.plain && whole && P.acc_out) {
            int32_t *ints = P.acc_out + at0;
#pragma unroll
            for (int i = 0; i < kAcc; ++i) {
                if (i * kStep >= left || !AXC_GLOBAL_OK(at0 + i * row + 3, (long long)g.M * g.Cout, 315u)) continue;
                const int a_code = P.acode ? P.a_coef * __ldg(P.acode + m0 + first + i * kStep) : 0;
                *reinterpret_cast<int4 *>(ints + i * row) = make_int4(acc[i][0] + back[0] + a_code, acc[i][1] + back[1] + a_code,
                                                                      acc[i][2] + back[2] + a_code, acc[i][3] + back[3] + a_code);
            }
        } else if (P.plain && whole) {
            // The common case on its own, in as few instructions as possible: the code is unrolled over the fragments and runs
            // once per tile, so its length is paid in instruction fetches (one loop for all cases: 51 000 clocks per tile of
            // 2048 pixels).  Four fragments at a time: what they read is requested before the first is finished.
            const float *asum = P.asum + (m0 + first), *res = P.residual + at0;
            float *out = P.output + at0;
            const int *acode = P.acode + (m0 + first);
#pragma unroll
            for (int i0 = 0; i0 < kAcc; i0 += EB) {
                float a_sum[EB];
                int a_code[EB];
                float4 r[EB];
#pragma unroll
                for (int i = 0; i < EB; ++i) a_code[i] = MODE == kXtabFull && P.acode && (i0 + i) * kStep < left ? P.a_coef * __ldg(acode + (i0 + i) * kStep) : 0;
#pragma unroll
                for (int i = 0; i < EB; ++i) a_sum[i] = (i0 + i) * kStep < left ? __fmul_rn(Q.m2, __ldg(asum + (i0 + i) * kStep)) : 0.0f;
                if (P.residual)
#pragma unroll
                    for (int i = 0; i < EB; ++i)
                        if ((i0 + i) * kStep < left) r[i] = __ldg(reinterpret_cast<const float4 *>(res + (i0 + i) * row));
#pragma unroll
                for (int i = 0; i < EB; ++i) {
                    float y[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        y[e] = __fsub_rn(__fadd_rn(__fadd_rn(__fmul_rn(float(acc[i0 + i][e] + back[e] + a_code[i]), Q.s1s2), a_sum[i]), t2[e]), Q.km1m2);
                    if (P.bias)
#pragma unroll
                        for (int e = 0; e < 4; ++e) y[e] = __fadd_rn(y[e], bias[e]);
                    if (P.residual) {
                        y[0] = __fadd_rn(y[0], r[i].x); y[1] = __fadd_rn(y[1], r[i].y);
                        y[2] = __fadd_rn(y[2], r[i].z); y[3] = __fadd_rn(y[3], r[i].w);
                    }
                    if ((i0 + i) * kStep < left && AXC_GLOBAL_OK(at0 + (i0 + i) * row + 3, (long long)g.M * g.Cout, 313u))
                        *reinterpret_cast<float4 *>(out + (i0 + i) * row) =
                            make_float4(max_keep_nan(y[0], P.out_floor), max_keep_nan(y[1], P.out_floor), max_keep_nan(y[2], P.out_floor), max_keep_nan(y[3], P.out_floor));
                }
            }
        } else {
#pragma unroll
            for (int i = 0; i < kAcc; ++i) {
                if (i * kStep >= left) continue;
                const long long at = at0 + i * row;
                if (!AXC_GLOBAL_OK(at, (long long)g.M * g.Cout, 314u)) continue;
                const float a_sum = P.partial ? 0.0f : __ldg(P.asum + m0 + first + i * kStep);
                const int a_code = P.acode && !P.partial ? P.a_coef * __ldg(P.acode + m0 + first + i * kStep) : 0;
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    if (j0 + e >= g.Cout) continue;
                    if (P.partial) {
                        if (!AXC_SCRATCH_OK(P, P.partial + at + e, 4, 342u)) continue;
                        atomicAdd(P.partial + at + e, acc[i][e]);
                        continue;
                    }
                    const int tot = acc[i][e] + back[e] + a_code;
                    float y = dequantise(Q, tot, a_sum, t2[e]);
                    if (P.bias) y = __fadd_rn(y, bias[e]);
                    if (P.residual) y = __fadd_rn(y, __ldg(P.residual + at + e));
                    if (P.output) P.output[at + e] = max_keep_nan(y, P.out_floor);
                    if (P.acc_out) P.acc_out[at + e] = tot;
                }
            }
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");               // nothing of this CTA is in flight when it ends
    if (!ok) {
        // thread 0 issued all bulk copies and, had every wait of its own come true, would have seen each of them arrive
        if (tid == 0) {
            if (kBuild) mbar_drain(rows_full, 0u);
            // tables asked for: all of this CTA's chunks, or as many as before the first wait that gave up
            const unsigned n = PRE ? min(chunk, lds32(asked)) : 0u;
            if (n > 1) mbar_drain(tab_full + (n & 1u) * 8, ((n - 2) >> 1) & 1u);
            if (n > 0) mbar_drain(tab_full + ((n - 1) & 1u) * 8, ((n - 1) >> 1) & 1u);
        }
        atomicExch(const_cast<int *>(&P.hdr->status), 3);
    }
}

// launch of a kernel that calls pdl_wait() before it touches what earlier kernels of the stream leave
template <typename Kernel, typename Params>
int launch_dependent(Kernel kernel, unsigned grid, unsigned threads, size_t smem, cudaStream_t stream, const Params &P)
{
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid); cfg.blockDim = dim3(threads); cfg.dynamicSmemBytes = smem; cfg.stream = stream;
    cfg.attrs = &attr; cfg.numAttrs = 1;
    AXC_CUDA(cudaLaunchKernelEx(&cfg, kernel, P));
    count_launch();
    return AXC_OK;
}

#include "axc_xref.cuh"

// The dequantisation of a call whose K was split over CTAs.
__global__ void __launch_bounds__(256) xfinal_kernel(const XParams P)
{
    pdl_trigger();
    pdl_wait();
    const DevQuant Q = *reinterpret_cast<const DevQuant *>(reinterpret_cast<const unsigned char *>(P.hdr) + kDevQuantOffset);
    // (at most 2^24 sums: kPartialMax)
    const unsigned total = unsigned(P.g.M) * unsigned(P.g.Cout), Cout = unsigned(P.g.Cout);
    auto one = [&](unsigned x, unsigned m, unsigned j, int sum, float a_sum, int a_code, float res) {
        const int tot = sum + P.k_e_min + a_code + (P.bcode ? P.b_coef * __ldg(P.bcode + j) : 0);
        float y = dequantise(Q, tot, a_sum, __fmul_rn(Q.m1, __ldg(P.bsum + j)));
        if (P.bias) y = __fadd_rn(y, __ldg(P.bias + j));
        if (P.residual) y = __fadd_rn(y, res);
        if (P.acc_out) P.acc_out[x] = tot;
        return max_keep_nan(y, P.out_floor);
    };
    const unsigned step = gridDim.x * 256u, first = blockIdx.x * 256u + threadIdx.x;
    if (Cout % 4 == 0 && ((reinterpret_cast<uintptr_t>(P.output) | reinterpret_cast<uintptr_t>(P.residual)) & 15u) == 0) {
        for (unsigned v = first; v < total / 4; v += step) {
            const unsigned x = v * 4, m = x / Cout, j = x - m * Cout;
            if (!AXC_SCRATCH_OK(P, P.partial + x, 16, 360u) || !AXC_SCRATCH_OK(P, P.asum + m, 4, 361u)) continue;
            const int4 sum = *reinterpret_cast<const int4 *>(P.partial + x);
            const float a_sum = __ldg(P.asum + m);
            const int a_code = P.acode ? P.a_coef * __ldg(P.acode + m) : 0;
            const float4 res = P.residual ? __ldg(reinterpret_cast<const float4 *>(P.residual + x)) : make_float4(0.f, 0.f, 0.f, 0.f);
            float4 y;
            y.x = one(x, m, j, sum.x, a_sum, a_code, res.x); y.y = one(x + 1, m, j + 1, sum.y, a_sum, a_code, res.y);
            y.z = one(x + 2, m, j + 2, sum.z, a_sum, a_code, res.z); y.w = one(x + 3, m, j + 3, sum.w, a_sum, a_code, res.w);
            if (P.output) *reinterpret_cast<float4 *>(P.output + x) = y;
        }
        return;
    }
    for (unsigned x = first; x < total; x += step) {
        const unsigned m = x / Cout, j = x - m * Cout;
        if (!AXC_SCRATCH_OK(P, P.partial + x, 4, 360u) || !AXC_SCRATCH_OK(P, P.asum + m, 4, 361u)) continue;
        const float y = one(x, m, j, P.partial[x], __ldg(P.asum + m), P.acode ? P.a_coef * __ldg(P.acode + m) : 0, P.residual ? __ldg(P.residual + x) : 0.0f);
        if (P.output) P.output[x] = y;
    }
}

// ------------------------------------------------------------------------------------------------------------------
// host
// ------------------------------------------------------------------------------------------------------------------
size_t r256(size_t v) { return (v + 255) & ~size_t(255); }

struct XLayout {
    size_t tt, wrow, wb, asum, bsum, acode, bcode, partial, codes, xt, xt_bytes, total;
};

constexpr size_t kPrepSmemMax = 220 * 1024;

struct PrepTile {
    int TH, TW, RH, RW, pitch, vec, bytes_at, bytes_pitch;
    size_t smem;
};

// Output pixels per preparation tile: at most one per thread, whatever is quickest by the clocks of a round: as many CTAs as shared
// memory and registers (two) allow, each loading its region (20 bytes per clock and SM, a batch of loads 700, a piece 100) and then
// adding K taps per pixel in a chain (4.5 clocks each, 32 taps per clock and SM at most).  Tiles of at most 72 KiB, as many as
// fill it, left 14 of 256 threads adding at 14x14x256.  Widths down to 7 pixels: without them 1x1 512 -> 128 at 28x28, 64 images, exact
// table, had tiles of 28 pixels in a row and took 113 us, with 7x7 95 (only where there are several rounds: else
// they gain nothing).  out == NULL: only whether there is such a tile.
bool prep_tile(const Geom &g, int vec, bool im2col, bool sums, PrepTile *out)
{
    PrepTile t = {};
    t.vec = vec;
    // an odd number of 16-byte pieces (floats) per pixel keeps the lanes of the patch sums on different banks
    if (vec) t.pitch = sums ? ((g.C >> 2) | 1) * 4 : 0;
    else t.pitch = im2col ? g.C : g.C | 1;
    auto region_h = [&](int th) { return size_t(th - 1) * g.sh + size_t(g.KH - 1) * g.dh + 1; };
    auto region_w = [&](int tw) { return size_t(tw - 1) * g.sw + size_t(g.KW - 1) * g.dw + 1; };
    // per pixel: the staged taps, then its code sum or (im2col) its codes - these not where one output pixel's region fills the
    // shared memory without them (a wide window with a wide dilation)
    bool bytes = im2col;
    auto smem = [&](size_t rh, size_t rw) { return (rh * rw * (size_t(t.pitch) * 4 + (bytes ? size_t(g.C) : im2col ? 0 : 4)) + (bytes ? 8 : 0) + 15) & ~size_t(15); };
    if (smem(region_h(1), region_w(1)) > kPrepSmemMax) bytes = false;
    if (smem(region_h(1), region_w(1)) > kPrepSmemMax) return false;
    if (!out) return true;
    double best = 1e300;
    const bool few = g.OW < 16 || g.M < 49 * 2 * kModelSms;        // one round whatever the tile
    for (int parts = 1, last = 0; !last; parts = parts < 4 ? parts + 1 : parts == 4 ? 7 : parts == 7 ? 8 : parts * 2) {
        last = parts >= g.OW;
        const int tw = last ? 1 : (g.OW + parts - 1) / parts;
        if (tw > kPrepThreads) continue;
        if (tw < 8 && g.OW >= 16 && best < 1e300 && (few || tw < 7)) break;      // (the search itself is host time of every call)
        if (parts == 7 && few) continue;
        const size_t rw = region_w(tw);
        for (int th = 1; th <= g.OH && th * tw <= kPrepThreads; th += th < 8 ? 1 : th < 16 ? 2 : 4) {
            const size_t rh = region_h(th), need = smem(rh, rw);
            if (need > kPrepSmemMax) break;
            const size_t block = (need < kSumSmem ? kSumSmem : need) + 1024;
            const int ctas = block * 2 <= 228 * 1024 ? 2 : 1;
            const long long tiles = (long long)g.N * ((g.OH + th - 1) / th) * ((g.OW + tw - 1) / tw), slots = kModelSms * ctas;
            const long long taps = (long long)rh * (long long)rw * g.C, per_batch = kPrepThreads * (vec ? 16 : 8);
            const double rounds = double((tiles + slots - 1) / slots);
            const double chain = sums ? 4.5 * g.K : 0.0, adds = sums ? double((th * tw + 31) / 32) * g.K : 0.0;
            const double load = double(taps) * 4.0 / 20.0;
            const double latency = 1000.0 + 700.0 * double((taps + per_batch - 1) / per_batch) + (vec ? 25.0 : 30.0) * double(taps / kPrepThreads);
            const double one = latency + chain, all = double(tiles) / kModelSms * (load + adds);
            const double cost = rounds * one > all ? rounds * one + 0.3 * all : all + 0.3 * rounds * one;
            if (cost < best) {
                best = cost;
                t.TH = th; t.TW = tw; t.RH = int(rh); t.RW = int(rw);
            }
        }
    }
    t.smem = smem(size_t(t.RH), size_t(t.RW));
    t.bytes_at = bytes ? t.RH * t.RW * t.pitch * 4 : -1;
    t.bytes_pitch = t.RW * g.C;
    if (t.smem < kSumSmem) t.smem = kSumSmem;
    *out = t;
    return true;
}

// Codes per pixel in 16-byte pieces, or im2col rows where the padding of the channel count to 16 would add more than an
// eighth to K.
void code_layout(const Geom &g, int *CC, int *chunks, int *im2col)
{
    const int cc = (g.C + 15) / 16, taps = g.KH * g.KW;
    const long long direct = (long long)taps * cc, rows = ((long long)g.K + 15) / 16;
    *im2col = direct * 8 > rows * 9 ? 1 : 0;
    *CC = *im2col ? int(rows) : cc;
    *chunks = int(*im2col ? rows : direct);
}

bool xgeom(const Geom &g, XGeom *x)
{
    if (g.M >= (1ll << 30) || (long long)g.N * g.H * g.W >= (1ll << 30)) return false;
    if (g.H >= 16384 || g.W >= 16384 || (long long)g.KH * g.dh >= 8192 || (long long)g.KW * g.dw >= 8192) return false;
    if ((long long)g.OH * g.sh >= 16384 || (long long)g.OW * g.sw >= 16384) return false;
    XGeom r;
    r.N = g.N; r.H = g.H; r.W = g.W; r.C = g.C; r.KH = g.KH; r.KW = g.KW; r.Cout = g.Cout;
    r.sh = g.sh; r.sw = g.sw; r.dh = g.dh; r.dw = g.dw; r.ph = g.ph; r.pw = g.pw; r.OH = g.OH; r.OW = g.OW; r.K = g.K; r.M = int(g.M);
    code_layout(g, &r.CC, &r.chunks, &r.im2col);
    const long long pieces = (r.im2col ? g.M : (long long)g.N * g.H * g.W) * r.CC;
    if (pieces >= (1ll << 29)) return false;      // word offsets of the codes fit an int
    // headroom for the piece number of a patch origin outside the image
    if (!r.im2col && (long long)(g.ph + g.KH * g.dh + 1) * g.W * r.CC >= (1ll << 29)) return false;
    r.TNC = 0; r.tiles_n = 0;
    *x = r;
    return true;
}

struct Config {
    int nb, splits, chunks_per_split;          // blocks of 8 pixels per warp; kXtabByte64: of a tile of 64 * nb pixels by two CTAs
    bool pre;
};

size_t xt_size(const XGeom &x, int mode) { return size_t((x.Cout + (mode == kXtabFull ? 7 : 15)) / (mode == kXtabFull ? 8 : 16)) * x.chunks * (mode == kXtabByte64 ? 16384u : 65536u); }

// Pixels per tile, splits of K, and where the expanded tables are made, by the clocks of all rounds (TileClocks below: per octet, lookups
// and codes per pixel, the waits around a table or building one; a start and an end; tables from global memory cost their writes and
// a launch).  Against every other tile, split and place forced (one B200, us per call, chosen / best / worst):
//   two digits                                        3x3 64 -> 96 at 28x28, 64 images    259 (1024, global) / 259 / 836
//                                                     3x3 64 -> 64 at 56x56, 64 images    679 (1024, global) / 660 (2048, global) / 2232
//   one byte, 256 rows (errors drawn from 0 .. 156)   3x3 512 -> 512 at 7x7, 1 image      126 (256, K in 9) / 126 / 1265
//                                                     3x3 64 -> 64 at 56x56, 1 image      28 (1024, K in 9, global) / 28 / 74
//                                                     3x3 64 -> 64 at 56x56, 8 images     69 (1024, global) / 69 / 176
//                                                     1x1 256 -> 1024 at 14x14, 8 images  56 (1024) / 56 / 119
//                                                     3x3 256 -> 256 at 14x14, 8 images   99 (2048, K in 9) / 99 / 384
//                                                     the same, 64 images                 451 (1024, K in 2, global) / 451 / 1221
//                                                     1x1 64 -> 256 at 56x56, 64 images   226 (1024, global) / 226 / 337
//                                                     1x1 1024 -> 2048 s2, 14x14, 64 im.  604 (2048) / 604 / 1120
//   exact products                                    3x3 512 -> 512 at 7x7, 1 image      51 (256, K in 9) / 51 / 202
//                                                     3x3 256 -> 256 at 14x14, 64 images  119 (2048) / 119 / 203
//                                                     3x3 192 -> 96 at 72x71, 12 images   171 (1024; K in 2 187) / 171 / 206
// Fitted over 74 layers each, 0.4 % (one byte) and 0.7 % (exact) above the best on average (0.8 % and 1.1 % over 40 drawn others); with the clocks of two-digit entries for
// all three it was 3.2 % and 2.4 %, up to 31 %.  A pixel of a 2048-pixel tile of bytes costs more (its registers spill), and so does a split
// of bytes: its sums are added one by one, and a pass over all of them follows.
// The same where the rows repeat: two CTAs of four warps to an SM, each with a half of a tile (of 2048 pixels: in two runs of 512,
// since 1024 pixels at a time have no registers left - 265 us against 222 on 1x1 64 -> 256 at 56x56, 64 images).  In clocks per octet of
// both CTAs: 2.18 per pixel of a half (also for a CTA that has the SM to itself, whose four warps wait for their loads), 250 for
// the waits around a table, 590 for building one.  Against all others forced (one B200, us per call, chosen / best / worst):
//   3x3 512 -> 512 at 7x7, 1 image                    70 (256, K in 9) / 70 / 1110
//   3x3 512 -> 512 at 7x7, 8 images                   103 (1024, K in 9) / 103 / 1139
//   1x1 512 -> 2048 at 7x7, 8 images                  55 (1024, K in 2) / 56 / 144
//   3x3 256 -> 256 at 14x14, 8 images                 90 (2048, K in 9, global) / 90 / 576
//   1x1 512 -> 128 at 28x28, 8 images                 45 (512, global) / 46 / 139
//   3x3 64 -> 64 at 56x56, 8 images                   66 (1024, K in 3, global) / 66 / 155
//   3x3 256 -> 256 at 14x14, 128 images               644 (1024, K in 3, global) / 644 / 1612
//   1x1 64 -> 256 at 56x56, 64 images                 232 (2048, global) / 232 / 559
//   3x3 32 -> 8 at 97x97, 20 images                   81 (2048, K in 3, global) / 76 (512, global) / 120
Config choose_halves(const XGeom &x, int sms, bool may_split, size_t xt_bytes)
{
    const int tiles_n = (x.Cout + 15) / 16, slots = 2 * sms;
    Config best = {16, 1, x.chunks, false};
    double best_cost = 1e300;
    for (int pre = 0; pre < 2; ++pre) {
        if (pre && xt_size(x, kXtabByte64) > xt_bytes) continue;
        for (int nb = 32; nb >= (pre ? 8 : 4); nb >>= 1) {
            const int group = nb == 32 ? 2 : 1, pix = 32 * nb / group;
            const long long tiles = ((long long)x.M + 32 * nb - 1) / (32 * nb) * tiles_n;
            // no split; as many as fill one to four rounds; two or three where there are rounds enough without and K is long
            const bool many = tiles >= slots;
            for (int r = 0; r <= 4; ++r) {
                if (r > 0 && (!may_split || (many && (r > 2 || x.chunks < 32)))) break;
                const long long fill = r == 0 ? 1 : many ? r + 1 : r * (long long)slots / tiles;
                const int sp = int(fill < x.chunks ? fill : x.chunks), cps = (x.chunks + sp - 1) / sp, spe = (x.chunks + cps - 1) / cps;
                const long long rounds = (tiles * spe + slots - 1) / slots;
                const double octet = 2.18 * pix + (pre ? 250.0 : 840.0), end = (pix == 512 ? 10.0 : 13.0) * pix;
                const double cost = double(rounds) * (group * (2.0 * cps * octet + end) + 2000.0) + (spe > 1 ? 7000.0 + double(x.M) * x.Cout / 300.0 : 0.0) +
                                    (pre ? double(xt_size(x, kXtabByte64)) / 1600.0 + 8600.0 : 3000.0);
                if (cost < best_cost) { best_cost = cost; best = {nb, spe, cps, pre != 0}; }
            }
        }
    }
    return best;
}

// Clocks of a tile: per pixel and octet of K (tiles of 4, 8, 16, 32 and 48 blocks per warp), around a table that comes from global
// memory or is built, a start, the end per pixel (plain / K split), a split's last pass and its sums, tables in global memory.
struct TileClocks {
    double pixel[5], copied, built, start, end, end_split, split, per_sum, tables, per_byte, own;
};
constexpr TileClocks kClocksFull = {{1.09, 1.09, 1.09, 1.09, 1.09}, 130, 850, 2000, 3.0, 6.0, 6000, 0.0, 8000, 1.0 / 2300, 3000};
constexpr TileClocks kClocksByte = {{1.13, 1.09, 1.055, 1.23, 0.0}, 110, 1010, 1000, 3.4, 16.0, 5500, 1.0 / 2150, 3150, 1.0 / 1430, 3000};
constexpr TileClocks kClocksExact = {{0.328, 0.30, 0.30, 0.333, 0.0}, 0, 118, 900, 5.6, 6.6, 2600, 1.0 / 356, 0, 0.0, 3000};

Config choose_config(int mode, const XGeom &x, int sms, bool may_split, size_t xt_bytes)
{
    if (mode == kXtabByte64) return choose_halves(x, sms, may_split, xt_bytes);
    const TileClocks &t = mode == kXtabFull ? kClocksFull : mode == kXtabByte ? kClocksByte : kClocksExact;
    const int tiles_n = (x.Cout + (mode == kXtabFull ? 7 : 15)) / (mode == kXtabFull ? 8 : 16);
    Config best = {32, 1, x.chunks, false};
    double best_cost = 1e300;
    for (int pre = 0; pre < 2; ++pre) {
        if (pre && (mode == kXtabExact || xt_size(x, mode) > xt_bytes)) continue;
        for (int nb = mode == kXtabFull && pre ? 48 : 32; nb >= (pre ? 16 : 4); nb = nb == 48 ? 32 : nb >> 1) {
            const int pix = kWarps * 8 * nb, size = nb == 48 ? 4 : nb == 32 ? 3 : nb == 16 ? 2 : nb == 8 ? 1 : 0;
            const long long tiles = ((long long)x.M + pix - 1) / pix * tiles_n;
            const double octet = t.pixel[size] * pix + (pre ? t.copied : t.built);
            // no split, or as many as fill one to four rounds; with bytes two or three where there are rounds enough without and K is long
            const bool many = tiles >= sms;
            for (int r = 0; r <= 4; ++r) {
                if (r > 0 && (!may_split || (many && (mode != kXtabByte || r > 2 || x.chunks < 32)))) break;
                const long long fill = r == 0 ? 1 : many ? r + 1 : r * (long long)sms / tiles;
                const int sp = int(fill < x.chunks ? fill : x.chunks);
                const int cps = (x.chunks + sp - 1) / sp;
                const int spe = (x.chunks + cps - 1) / cps;
                const long long rounds = (tiles * spe + sms - 1) / sms;
                double cost = double(rounds) * (2.0 * cps * octet + t.start + pix * (spe > 1 ? t.end_split : t.end)) + (spe > 1 ? t.split + double(x.M) * x.Cout * t.per_sum : 0.0);
                cost += pre ? double(xt_size(x, mode)) * t.per_byte + t.tables : t.own;
                if (cost < best_cost) { best_cost = cost; best = {nb, spe, cps, pre != 0}; }
            }
        }
    }
    return best;
}

XLayout xlayout(const Geom &g, const XGeom &x, int mode)
{
    XLayout L;
    const size_t cout16 = size_t((g.Cout + 15) / 16) * 16;
    size_t off = 256;
    L.tt = off;      off += r256(257 * 512);
    L.wrow = off;    off += r256(cout16 * x.chunks * 32);
    L.wb = off;      off += r256(cout16 * x.chunks * 16);
    L.asum = off;    off += r256(size_t(g.M) * 4);
    L.bsum = off;    off += r256(size_t(g.Cout) * 4);
    L.acode = off;   off += r256(size_t(g.M) * 4);
    L.bcode = off;   off += r256(size_t(g.Cout) * 4);
    L.partial = off; off += r256(size_t(g.M) * g.Cout * 4 <= kPartialMax && mode != kXtabRef ? size_t(g.M) * g.Cout * 4 : 0);
    L.codes = off;   off += r256((x.im2col ? size_t(g.M) : size_t(g.N) * g.H * g.W) * x.CC * 16);
    // room for the expanded tables where a call would have them made in global memory
    L.xt = off;
    L.xt_bytes = 0;
    for (int m : {int(kXtabByte), int(kXtabByte64), int(kXtabFull)}) {
        const size_t bytes = xt_size(x, m);
        if ((mode == m || mode == kXtabAny) && bytes <= kXtMax && bytes > L.xt_bytes && choose_config(m, x, kModelSms, size_t(g.M) * g.Cout * 4 <= kPartialMax, bytes).pre) L.xt_bytes = bytes;
    }
    off += L.xt_bytes;
    L.total = off;
    return L;
}

template <int MODE, int NB, bool PRE>
int launch_variant(const XParams &P, const DeviceInfo &di, cudaStream_t stream)
{
    constexpr bool kHalf = MODE == kXtabByte64;                    // two CTAs to an SM, each a half of the tiles
    const int smem = kHalf ? int(kWindowHalf - di.smem_base) : di.max_smem_optin, slots = kHalf ? 2 * di.sm_count : di.sm_count;
    AXC_CUDA(cudaFuncSetAttribute(xtab_kernel<MODE, NB, PRE>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    const long long turns = kHalf ? P.units / P.group : P.units, grid = turns < slots ? turns : slots;
    return launch_dependent(xtab_kernel<MODE, NB, PRE>, unsigned(grid), kWarpsOf<MODE> * 32, size_t(smem), stream, P);
}

template <int MODE>
int launch_mode(const Config &cf, const XParams &P, const DeviceInfo &di, cudaStream_t stream)
{
    constexpr bool kPre = MODE != kXtabExact;
    if (cf.pre) {
        if (cf.nb == 48) return launch_variant<MODE, MODE == kXtabFull ? 48 : 16, kPre>(P, di, stream);
        if (cf.nb == 8) return launch_variant<MODE, MODE == kXtabByte64 ? 8 : 16, kPre>(P, di, stream);
        return cf.nb == 32 && MODE != kXtabByte64 ? launch_variant<MODE, MODE == kXtabByte64 ? 16 : 32, kPre>(P, di, stream) : launch_variant<MODE, 16, kPre>(P, di, stream);
    }
    switch (cf.nb) {
    case 32: return launch_variant<MODE, MODE == kXtabByte64 ? 16 : 32, false>(P, di, stream);
    case 16: return launch_variant<MODE, 16, false>(P, di, stream);
    case 8: return launch_variant<MODE, 8, false>(P, di, stream);
    default: return launch_variant<MODE, 4, false>(P, di, stream);
    }
}

template <int MODE>
int launch_expand(const ExpandParams &E, const DeviceInfo &di, cudaStream_t stream)
{
    constexpr size_t smem = MODE == kXtabFull ? 257 * 512 + 2 * 16 * 8 * 2 + 16 : 257 * (MODE == kXtabByte ? 256 : 128) + (MODE == kXtabByte ? 2 : 4) * 16 * 16 * 2 + 16;
    AXC_CUDA(cudaFuncSetAttribute(xexpand_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
    const int total = E.g.tiles_n * E.g.chunks, turns = MODE == kXtabByte64 ? (total + 1) / 2 : total, slots = di.sm_count * (MODE == kXtabByte64 ? 2 : 1);
    const int grid = turns < slots ? turns : slots;
    return launch_dependent(xexpand_kernel<MODE>, unsigned(grid), kExpandThreads, smem, stream, E);
}

}  // namespace

size_t xtab_scratch_bytes(const Geom &g, int mode)
{
    if (mode == kXtabNone) return 0;
    // Calls with fewer lookups stay on the plan-based kernels.  The line is a cautious one, not the crossing: measured with it at 0
    // (us per call, a filter whose plan is kept / expanded tables; CUDA-graph replay in brackets), the expanded tables are faster at
    // every size tried - 50 / 31 (41 / 14) at 3.0e5 lookups, 69 / 31 (59 / 16) at 1.8e6, 40 / 26 (31 / 18) at 6.4e6,
    // 104 / 31 (94 / 25) at 1.5e7 - and a new filter's plan costs 1.2 to 22 ms on top.
    if ((double)g.M * g.K * g.Cout < kXtabMinLookups) return 0;
    XGeom x;
    if (!xgeom(g, &x) || !prep_tile(g, g.C % 4 == 0 && !x.im2col, x.im2col != 0, true, nullptr) || !prep_tile(g, 0, x.im2col != 0, true, nullptr)) return 0;
    return xlayout(g, x, mode).total;
}

bool xtab_ref_pays(const Geom &g)
{
    XGeom x;
    return xgeom(g, &x) && xref_pays(x);
}

void xtab_config(const Geom &g, int mode, int32_t out3[3])
{
    XGeom x;
    xgeom(g, &x);
    if (mode == kXtabRef) {
        out3[0] = xref_tile(x, kModelSms); out3[1] = 1; out3[2] = 0;
        return;
    }
    const Config cf = choose_config(mode, x, kModelSms, size_t(g.M) * g.Cout * 4 <= kPartialMax, xlayout(g, x, mode).xt_bytes);
    out3[0] = kWarps * 8 * cf.nb; out3[1] = cf.splits; out3[2] = cf.pre ? 1 : 0;
}

int launch_xtab(const uint16_t *lut_dev, int mode, int centred, int e_min, const Geom &g, const Quant &q, const float *ranges_dev,
                const float *input, const float *filter, float *output, unsigned char *scratch, const axc_debug_out *dbg,
                const DeviceInfo &di, cudaStream_t stream, const QuantisedOperands *u8)
{
    PrepParams A;
    XParams P;
    if (!xgeom(g, &A.g)) return AXC_INTERNAL;
    XGeom &x = A.g;
    x.TNC = two_bytes(mode) ? 8 : 16;
    x.tiles_n = (g.Cout + x.TNC - 1) / x.TNC;
    const XLayout L = xlayout(g, x, mode);
    const size_t partial_bytes = size_t(g.M) * g.Cout * 4;
    const Config cf = mode == kXtabRef ? Config{0, 1, x.chunks, false} : choose_config(mode, x, di.sm_count, partial_bytes <= kPartialMax, L.xt_bytes);
    const int vec = (g.C % 4 == 0 && !x.im2col && (u8 ? (reinterpret_cast<uintptr_t>(u8->input) & 3u) : (reinterpret_cast<uintptr_t>(input) & 15u)) == 0) ? 1 : 0;
    PrepTile t;
    A.sums = u8 ? 0 : 1;
    if (!prep_tile(g, vec, x.im2col != 0, A.sums != 0, &t)) return AXC_INTERNAL;
    A.input_u8 = u8 ? u8->input : nullptr; A.filter_u8 = u8 ? u8->filter : nullptr; A.pad = u8 ? u8->input_offset & 255 : 0;
    A.input = input; A.filter = filter; A.lut = lut_dev; A.ranges = ranges_dev; A.host_q = host_dev_quant(q, g.K);
    A.in_floor = g.ep.input_relu ? 0.0f : -INFINITY;
    A.mode = mode; A.centred = centred; A.e_min = e_min;
    P.a_coef = 128 * centred - (u8 ? u8->filter_offset : 0);
    P.b_coef = 128 * centred - (u8 ? u8->input_offset : 0);
    const bool sums = P.a_coef != 0 || P.b_coef != 0;
    A.acode = sums ? reinterpret_cast<int *>(scratch + L.acode) : nullptr;
    A.bcode = sums ? reinterpret_cast<int *>(scratch + L.bcode) : nullptr;
    A.codes = scratch + L.codes; A.tt = scratch + L.tt;
    A.wrow = reinterpret_cast<uint16_t *>(scratch + L.wrow); A.wb = reinterpret_cast<uint2 *>(scratch + L.wb);
    A.asum = reinterpret_cast<float *>(scratch + L.asum); A.bsum = reinterpret_cast<float *>(scratch + L.bsum);
    A.qf_debug = dbg ? dbg->qfilter : nullptr;
    A.hdr = reinterpret_cast<PlanHeader *>(scratch);
    A.scratch_bytes = P.scratch_bytes = (long long)L.total;
    A.TH = t.TH; A.TW = t.TW; A.RH = t.RH; A.RW = t.RW; A.pitch = t.pitch; A.vec = t.vec; A.bytes_at = t.bytes_at; A.bytes_pitch = t.bytes_pitch;
    A.tiles_y = (g.OH + t.TH - 1) / t.TH; A.tiles_x = (g.OW + t.TW - 1) / t.TW;
    A.blocks_sum = A.sums || A.bcode ? (g.Cout + 31) / 32 : 0;
    const long long w_warps = (long long)x.tiles_n * x.chunks;
    A.blocks_w = cf.pre ? 0 : int((w_warps + 15) / 16 < 296 ? (w_warps + 15) / 16 : 296);
    A.blocks_t = cf.pre || mode == kXtabExact ? 0 : 32;
    const long long blocks = (long long)A.blocks_sum + A.blocks_w + A.blocks_t + (long long)g.N * A.tiles_y * A.tiles_x;
    if (blocks >= (1ll << 31)) return AXC_INTERNAL;
    P.partial = nullptr;
    A.zeros = nullptr; A.zero_pieces = 0;
    if (cf.splits > 1) {
        P.partial = reinterpret_cast<int32_t *>(scratch + L.partial);
        A.zeros = reinterpret_cast<uint4 *>(P.partial);
        A.zero_pieces = (long long)((partial_bytes + 15) / 16);    // (the region is rounded up to 256 bytes)
    }
    const auto prep = u8 ? xprep_kernel<true> : xprep_kernel<false>;
    AXC_CUDA(cudaFuncSetAttribute(prep, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kPrepSmemMax)));
    // An SM that runs preparation CTAs is asked for all of its shared memory.  With no more than those need the CTAs of the kernels
    // behind, launched while these run, find no room beside them and wait until the SM is empty: 1x1 64 -> 64 at 56x56, 8 images,
    // 256-row tables 22.7 us per call, so 18.6; 1 % over 309 layers and forms.
    cudaLaunchAttribute carveout;
    carveout.id = cudaLaunchAttributePreferredSharedMemoryCarveout;
    carveout.val.sharedMemCarveout = cudaSharedmemCarveoutMaxShared;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(unsigned(blocks)); cfg.blockDim = dim3(kPrepThreads); cfg.dynamicSmemBytes = t.smem; cfg.stream = stream;
    cfg.attrs = &carveout; cfg.numAttrs = 1;
    AXC_CUDA(cudaLaunchKernelEx(&cfg, prep, A));
    count_launch();

    if (cf.pre) {
        ExpandParams E;
        E.g = x; E.filter = filter; E.filter_u8 = A.filter_u8; E.rows = reinterpret_cast<const unsigned char *>(lut_dev + 65536); E.ranges = ranges_dev; E.host_q = A.host_q;
        E.xt = scratch + L.xt; E.wb = A.wb; E.qf_debug = A.qf_debug; E.hdr = A.hdr; E.scratch_bytes = A.scratch_bytes;
        const int rc = mode == kXtabFull ? launch_expand<kXtabFull>(E, di, stream) : mode == kXtabByte ? launch_expand<kXtabByte>(E, di, stream) : launch_expand<kXtabByte64>(E, di, stream);
        if (rc) return rc;
    }

    P.g = x;
    P.xt = cf.pre ? scratch + L.xt : nullptr;
    P.codes = A.codes; P.tt = A.tt; P.wrow = A.wrow; P.wb = A.wb; P.asum = A.asum; P.bsum = A.bsum; P.hdr = A.hdr;
    P.output = output; P.acc_out = dbg ? dbg->acc : nullptr;
    P.acode = A.acode; P.bcode = A.bcode;
    P.bias = g.ep.bias; P.residual = g.ep.residual; P.out_floor = g.ep.relu ? 0.0f : -INFINITY;
    P.k_e_min = int(unsigned(g.K) * (unsigned(e_min) + (u8 ? unsigned(u8->input_offset) * unsigned(u8->filter_offset) : 0u)));
    if (mode == kXtabRef) return launch_ref(P, di, stream);
    P.splits = cf.splits; P.chunks_per_split = cf.chunks_per_split;
    const int tile = (mode == kXtabByte64 ? kWarpsOf<kXtabByte64> : kWarps) * 8 * cf.nb;
    P.group = mode == kXtabByte64 && cf.nb == 32 ? 2 : 1;
    P.units = ((long long)x.M + tile - 1) / tile * x.tiles_n * cf.splits * P.group;
    if (P.units >= (1ll << 31)) return AXC_INTERNAL;
    P.plain = ((output != nullptr) != (P.acc_out != nullptr) && !P.partial &&
               ((reinterpret_cast<uintptr_t>(output) | reinterpret_cast<uintptr_t>(P.acc_out) | reinterpret_cast<uintptr_t>(g.ep.residual)) & 15u) == 0) ? 1 : 0;
    int rc = mode == kXtabFull ? launch_mode<kXtabFull>(cf, P, di, stream)
             : mode == kXtabByte ? launch_mode<kXtabByte>(cf, P, di, stream)
             : mode == kXtabByte64 ? launch_mode<kXtabByte64>(cf, P, di, stream) : launch_mode<kXtabExact>(cf, P, di, stream);
    if (rc) return rc;
    if (cf.splits > 1) {
        const long long n = (g.M * g.Cout + (g.Cout % 4 == 0 ? 1023 : 255)) / (g.Cout % 4 == 0 ? 1024 : 256);
        return launch_dependent(xfinal_kernel, unsigned(n < 1184 ? n : 1184), 256, 0, stream, P);
    }
    return AXC_OK;
}

AXC_DEFINE_BOUNDS_READER(bounds_record_xtab)

#ifdef AXC_BOUNDS_CHECK
int set_wait_polls(int expand, int convolution)
{
    const int polls[2] = {expand < 0 ? kWaitPolls : expand, convolution < 0 ? kWaitPolls : convolution};
    AXC_CUDA(cudaMemcpyToSymbol(g_wait_polls, polls, sizeof(polls)));
    return AXC_OK;
}
#endif

}  // namespace axc

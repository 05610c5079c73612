// The reference's order of additions on expanded tables (included by axc_xtab.cu): an fp32 running total that takes the looked-up
// entries one by one in K order (tf2/src/approx_nn_conv_kernels.cpp:245-246, 201-202).
//
// A lane owns a pixel and the totals of 8 channels: one LDS.128 returns the 8 entries of a K element.  All lanes must walk K from
// its start, so the 8 lanes of a quarter warp cannot take 8 different elements at once as in xtab_kernel; instead lane d runs d
// elements behind: at step s it looks element s - d up, and the quarter warp reads 8 different 16-byte bank groups whatever
// the codes are.  The window of live elements is 8 long, so the expanded table is a ring of 16 elements (64 KiB) that is built
// four at a time, one group ahead.  The lag costs a byte rotation of the codes per 16 elements and 8 steps per tile.
//
// An entry v < 2^16 is, as loaded, the bits of the fp32 subnormal v * 2^-149: total = fma(entry, 2^125, total) adds v * 2^-24 with
// one rounding, and a total kept less 24 binary places rounds exactly where the reference's does (fp32 multiples of 2^-24 below
// 2^8).  Two channels per FMA (f32x2); what is left per lookup is half an instruction, one to take the entry out of its
// word, and an eighth of address and load.
//
// Bound: shared memory, one clock per pixel and element of a tile for the lookups and 96 for the building (per element and 8
// channels 32 clocks of reads and 64 of writes, which reach only 4 of the 8 bank groups), next to as many clocks of issue.
// 3x3 256 -> 256 at 14x14, 16 images: 508 us per call, against 877 of lookups of one entry per lane with bank conflicts
// (dense_kernel<WN, true>).

constexpr int kRefThreads = 512, kRefWarps = kRefThreads / 32;

struct RefParams {
    XParams x;
    int tile;                   // output pixels per unit, a multiple of 32
};

__device__ __forceinline__ void add_entries(unsigned long long &total, unsigned word)
{
    // channels 2i and 2i + 1: low and high half of the word
    const unsigned long long entries = (unsigned long long)(word >> 16) << 32 | (word & 0xFFFFu);
    const unsigned long long scale = 0x7E0000007E000000ull;          // 2^125, twice
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(total) : "l"(entries), "l"(scale));
}

template <int PXL>
__global__ void __launch_bounds__(kRefThreads, 1) xref_kernel(const RefParams R)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const XParams &P = R.x;
    const XGeom &g = P.g;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned dyn0 = (unsigned)__cvta_generic_to_shared(smem_raw);
    unsigned dyn_size;
    asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dyn_size));
    const unsigned rows_full = (dyn0 + 15u) & ~15u;
    pdl_wait();
    if (rows_full + 8u > kCodes || dyn0 + dyn_size < kWindowEnd) {
        if (tid == 0) atomicExch(const_cast<int *>(&P.hdr->status), 2);
        return;
    }
    if (tid == 0) {
        mbar_init(rows_full, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(rows_full), "r"(257u * 512u) : "memory");
        bulk_copy(kRowsLow, P.tt, kLowRows * 512u, rows_full);
        bulk_copy(kRowsHigh, P.tt + kLowRows * 512u, (257u - kLowRows) * 512u, rows_full);
    }
    __syncthreads();
    bool ok = true;
    mbar_wait(rows_full, 0u, ok, AXC_WAIT_POLLS(1));

    const DevQuant Q = *reinterpret_cast<const DevQuant *>(reinterpret_cast<const unsigned char *>(P.hdr) + kDevQuantOffset);
    const int pieces = g.im2col ? g.M : g.N * g.H * g.W;           // distance of the 16-byte pieces of one pixel
    const int eh = g.im2col ? 1 : g.H, ew = g.im2col ? 1 : g.W;
    const unsigned d = unsigned(lane & 7), db = (d & 3u) * 8u;      // how far the lane lags, and its odd bytes in bits
    unsigned row_of[16];                                           // step s: where the ring's row 0 has element s - d
#pragma unroll
    for (unsigned s = 0; s < 16; ++s) row_of[s] = kTab + (((s - d) & 15u) << 4);

    // ---- building: a lane takes one word (two a) of the rows of one element's 8 weights and writes the pieces of those a ----------
    const unsigned kidx = unsigned(lane & 3), sub = unsigned(lane >> 2);
    const unsigned word = unsigned(warp >> 2) * 32u + ((8u * (unsigned(warp & 3) + kidx) + sub) & 31u);
    unsigned raw[8];
    auto build_load = [&](const uint4 &list) {
        const unsigned l4[4] = {list.x, list.y, list.z, list.w};
#pragma unroll
        for (int s = 0; s < 8; ++s) raw[s] = lds32(((s & 1) ? l4[s >> 1] >> 16 : l4[s >> 1] & 0xFFFFu) * 16u + word * 4u);
    };
    auto build_store = [&](unsigned group) {
        const unsigned dst = kTab + word * 512u + (((group & 3u) * 4u + kidx) << 4);
        sts128(dst, make_uint4(prmt<0x5410>(raw[0], raw[1]), prmt<0x5410>(raw[2], raw[3]), prmt<0x5410>(raw[4], raw[5]), prmt<0x5410>(raw[6], raw[7])));
        sts128(dst + 256u, make_uint4(prmt<0x7632>(raw[0], raw[1]), prmt<0x7632>(raw[2], raw[3]), prmt<0x7632>(raw[4], raw[5]), prmt<0x7632>(raw[6], raw[7])));
    };
    const int groups = g.chunks * 4;
    constexpr unsigned kNullRow = (kRowsHigh + (unsigned(kNull) - kLowRows) * 512u) >> 4;
    const uint4 nothing = make_uint4(kNullRow * 0x10001u, kNullRow * 0x10001u, kNullRow * 0x10001u, kNullRow * 0x10001u);

    for (unsigned u = blockIdx.x; u < unsigned(P.units); u += gridDim.x) {
        const int mt = int(u / unsigned(g.tiles_n)), nt = int(u - unsigned(mt) * unsigned(g.tiles_n));
        const int m0 = mt * R.tile;
        const uint4 *lists = reinterpret_cast<const uint4 *>(P.wrow) + (size_t)nt * g.chunks * 16 + kidx;
        auto list_of = [&](int q) { return q < groups && AXC_SCRATCH_OK(P, lists + q * 4, 16, 371u) ? __ldg(lists + q * 4) : nothing; };
        // the lane's pixels: 32 neighbouring ones per warp, the warps in turn
        int base[PXL], yx[PXL];
#pragma unroll
        for (int i = 0; i < PXL; ++i) {
            const int p = (i * kRefWarps + warp) * 32 + lane, m = m0 + p;
            base[i] = 0; yx[i] = -32768 * 65536;                   // no pixel: every tap out of range
            if (p < R.tile && m < g.M) {
                int y = 0, x = 0, b = m;
                if (!g.im2col) {
                    const unsigned mm = unsigned(m), row = mm / unsigned(g.OW), n = row / unsigned(g.OH);
                    y = int(row - n * unsigned(g.OH)) * g.sh - g.ph;
                    x = int(mm - row * unsigned(g.OW)) * g.sw - g.pw;
                    b = (int(n) * g.H + y) * g.W + x;
                }
                base[i] = b;
                yx[i] = (y << 16) | (x & 0xFFFF);
            }
        }
        int used = 0;                                              // pixels of this warp that exist (the same for all lanes)
#pragma unroll
        for (int i = 0; i < PXL; ++i) used += (i * kRefWarps + warp) * 32 < R.tile && m0 + (i * kRefWarps + warp) * 32 < g.M ? 1 : 0;
        int f_cc = 0, f_kx = 0, f_ky = 0;
        uint4 next[PXL];
        auto fetch = [&]() {                                       // the next chunk's codes of the lane's pixels
            const int dy = f_ky * g.dh, dx = f_kx * g.dw, off = dy * g.W + dx + f_cc * pieces;
#pragma unroll
            for (int i = 0; i < PXL; ++i) {
                const bool in = unsigned((yx[i] >> 16) + dy) < unsigned(eh) && unsigned(int(short(yx[i])) + dx) < unsigned(ew) &&
                                AXC_GLOBAL_OK(base[i] + off, (long long)pieces * g.CC, 372u);
                next[i] = in ? __ldg(reinterpret_cast<const uint4 *>(P.codes) + unsigned(base[i] + off)) : make_uint4(0, 0, 0, 0);
            }
            if (++f_cc == g.CC && !g.im2col) { f_cc = 0; if (++f_kx == g.KW) { f_kx = 0; ++f_ky; } }
        };

        unsigned long long total[PXL][4];
        unsigned last[PXL][2];                                     // the last 8 codes of the chunk before
#pragma unroll
        for (int i = 0; i < PXL; ++i) {
#pragma unroll
            for (int e = 0; e < 4; ++e) total[i][e] = 0;
            last[i][0] = last[i][1] = 0;
        }
        fetch();
        // the elements before the first (slots 8..15) are all zeros, then the first group
        build_load(nothing);
        build_store(2); build_store(3);
        build_load(list_of(0));
        build_store(0);
        uint4 list = list_of(1);
        __syncthreads();
        for (int c = 0; c <= g.chunks; ++c) {
            unsigned code[PXL][4];                                 // 16 codes, the lane's lag behind the chunk
#pragma unroll
            for (int i = 0; i < PXL; ++i) {
                const unsigned w[6] = {last[i][0], last[i][1], next[i].x, next[i].y, next[i].z, next[i].w};
                unsigned v[5];
#pragma unroll
                for (int e = 0; e < 5; ++e) v[e] = d >= 4u ? w[e] : w[e + 1];
#pragma unroll
                for (int e = 0; e < 4; ++e) code[i][e] = __funnelshift_l(v[e], v[e + 1], db);
                last[i][0] = next[i].z; last[i][1] = next[i].w;
            }
            // after the last chunk the lagging lanes have 7 elements to go, the others look zeros up
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                const int q = c * 4 + h;
                if (q >= groups + 2) break;
                // (loads and stores keep this order: lookups of two steps in flight, the building between them)
                constexpr unsigned kSel[4] = {0x3240u, 0x3250u, 0x3260u, 0x3270u};          // {low byte, code, upper half}
                uint4 x[2][PXL];
                auto look = [&](int j) {
#pragma unroll
                    for (int i = 0; i < PXL; ++i)
                        if (i < used) x[j & 1][i] = lds128(prmt_r(row_of[h * 4 + j], code[i][h], kSel[j]));
                };
                auto add = [&](int j) {
#pragma unroll
                    for (int i = 0; i < PXL; ++i)
                        if (i < used) {
                            const uint4 &v = x[j & 1][i];
                            add_entries(total[i][0], v.x); add_entries(total[i][1], v.y);
                            add_entries(total[i][2], v.z); add_entries(total[i][3], v.w);
                        }
                };
                look(0);
                build_load(list);
                list = list_of(q + 2);
                if (h == 3 && c + 1 < g.chunks) fetch();
                if (h == 3 && c + 1 >= g.chunks)
#pragma unroll
                    for (int i = 0; i < PXL; ++i) next[i] = make_uint4(0, 0, 0, 0);
                look(1);
                add(0);
                build_store(unsigned(q + 1));
                look(2);
                add(1);
                look(3);
                add(2);
                add(3);
                __syncthreads();                                   // group q + 1 is there, group q - 2 is done with
            }
        }
        // ---- dequantise and store: 8 neighbouring channels of a pixel ------------------------------------------------------
        const int j0 = nt * 8;
#pragma unroll
        for (int i = 0; i < PXL; ++i) {
            const int p = (i * kRefWarps + warp) * 32 + lane, m = m0 + p;
            if (p >= R.tile || m >= g.M || !AXC_SCRATCH_OK(P, P.asum + m, 4, 373u)) continue;
            const float a_sum = __ldg(P.asum + m);
            const long long at = (long long)m * g.Cout + j0;
            float y[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                y[e] = 0.0f;
                if (j0 + e >= g.Cout || !AXC_GLOBAL_OK(at + e, (long long)g.M * g.Cout, 374u)) continue;
                const float sum = __fmul_rn(__uint_as_float(unsigned(total[i][e >> 1] >> ((e & 1) * 32))), 16777216.0f);
                y[e] = __fsub_rn(__fadd_rn(__fadd_rn(__fmul_rn(sum, Q.s1s2), __fmul_rn(Q.m2, a_sum)), __fmul_rn(Q.m1, __ldg(P.bsum + j0 + e))), Q.km1m2);
                if (P.bias) y[e] = __fadd_rn(y[e], __ldg(P.bias + j0 + e));
                if (P.residual) y[e] = __fadd_rn(y[e], __ldg(P.residual + at + e));
                y[e] = max_keep_nan(y[e], P.out_floor);
                if (P.acc_out) P.acc_out[at + e] = __float2int_rz(sum);
            }
            if (P.plain && j0 + 8 <= g.Cout && AXC_GLOBAL_OK(at + 7, (long long)g.M * g.Cout, 375u)) {
                *reinterpret_cast<float4 *>(P.output + at) = make_float4(y[0], y[1], y[2], y[3]);
                *reinterpret_cast<float4 *>(P.output + at + 4) = make_float4(y[4], y[5], y[6], y[7]);
            } else {
#pragma unroll
                for (int e = 0; e < 8; ++e)
                    if (j0 + e < g.Cout && AXC_GLOBAL_OK(at + e, (long long)g.M * g.Cout, 376u)) P.output[at + e] = y[e];
            }
        }
    }
    if (!ok) {
        if (tid == 0) mbar_drain(rows_full, 0u);
        atomicExch(const_cast<int *>(&P.hdr->status), 3);
    }
}

// Pixels per tile: a multiple of 32 up to 2048 that shares the pixels evenly, by the clocks of all rounds - per octet of K one
// clock per pixel and element for the lookups, 1.4 with what the issue slots add, 850 for the building and its barriers.
int xref_tile(const XGeom &x, int sms)
{
    const int tiles_n = (x.Cout + 7) / 8;
    int best = 2048;
    double best_cost = 1e300;
    for (int n = 1; n <= 4096; n = n < 64 ? n + 1 : n * 2) {
        const long long share = ((long long)x.M + n - 1) / n;
        const int tile = share >= 2048 ? 2048 : int((share + 31) / 32 * 32);
        const long long units = ((long long)x.M + tile - 1) / tile * tiles_n, rounds = (units + sms - 1) / sms;
        const double cost = double(rounds) * ((2.0 * x.chunks + 1.0) * (1.4 * tile + 850.0) + 3000.0 + 4.0 * tile);
        if (cost < best_cost) { best_cost = cost; best = tile; }
        if (tile <= 128) break;
    }
    return best;
}

// The other kernel for this order (dense_kernel<WN, true>: a tile of 64 pixels x 64 channels, or 128 x 32, per SM and round) goes round
// less often where there are few pixels and many channels.  In us, fitted to 57 layers (within 16 %, the other within 10 % from
// K = 256 on), 148 SMs; expanded tables / the other, measured:
//   1x1 2048 -> 4096, one pixel             889 / 405    (4 rounds / 1)        1x1 2048 -> 512 at 7x7, 4 images       252 / 409    (1 / 1)
//   1x1 512 -> 2048 at 7x7, 4 images        137 / 111    (2 / 1)               1x1 512 -> 2048 at 7x7, 16 images      242 / 293    (2 / 3)
//   1x1 1024 -> 2048 s2 at 14x14, 4 images  270 / 214    (2 / 1)               3x3 256 -> 256 at 14x14, 16 images     506 / 862    (1 / 2)
bool xref_pays(const XGeom &x)
{
    constexpr long long sms = kModelSms;
    const long long tile = xref_tile(x, kModelSms), units = (x.M + tile - 1) / tile * ((x.Cout + 7) / 8), rounds = (units + sms - 1) / sms;
    const int tn = x.Cout <= 32 ? 32 : 64, tm = 4096 / tn;
    const long long others = (x.M + tm - 1ll) / tm * ((x.Cout + tn - 1) / tn), other_rounds = (others + sms - 1) / sms;
    return double(rounds) * ((2.0 * x.chunks + 1.0) * (0.86 + 0.0011 * double(tile)) + 0.0136 * double(tile)) <= x.K * (0.172 * double(other_rounds) + 0.033);
}

template <int PXL>
int launch_ref_variant(const RefParams &R, const DeviceInfo &di, cudaStream_t stream)
{
    AXC_CUDA(cudaFuncSetAttribute(xref_kernel<PXL>, cudaFuncAttributeMaxDynamicSharedMemorySize, di.max_smem_optin));
    const long long grid = R.x.units < di.sm_count ? R.x.units : di.sm_count;
    return launch_dependent(xref_kernel<PXL>, unsigned(grid), kRefThreads, size_t(di.max_smem_optin), stream, R);
}

int launch_ref(XParams &P, const DeviceInfo &di, cudaStream_t stream)
{
    RefParams R;
    R.tile = xref_tile(P.g, di.sm_count);
    P.units = ((long long)P.g.M + R.tile - 1) / R.tile * P.g.tiles_n;
    if (P.units >= (1ll << 31)) return AXC_INTERNAL;
    P.plain = ((reinterpret_cast<uintptr_t>(P.output) & 15u) == 0 && P.g.Cout % 4 == 0) ? 1 : 0;
    R.x = P;
    const int pixels = kRefThreads;
    return R.tile <= pixels ? launch_ref_variant<1>(R, di, stream) : R.tile <= 2 * pixels ? launch_ref_variant<2>(R, di, stream)
           : R.tile <= 3 * pixels ? launch_ref_variant<3>(R, di, stream) : launch_ref_variant<4>(R, di, stream);
}

// Half-precision convolutions as implicit products on tcgen05: forward, input gradient and weight gradient of layers with enough work
// (px_pays, px_wg_pays), any plane size and channel count, windows of up to 49 taps, strides of up to 3.
// [ref: lib/sources/pulp_conv2d_fp32.c:85-113 (FW), :294-333 (WG), :504-549 (IG); naive kernels pulp_conv_naive_fp32.c:198-516]
//
// The planes of all streams are laid end to end as SLOTS: row after row, a row longer than the image by as many zero slots as
// the window reaches past it, a plane by as many zero rows.  The zeros behind one row serve as the padding in front of the
// next, so 28 x 28 pixels with a 3 x 3 window take 29 x 29 slots.  A filter tap is then one fixed distance in slots, for every
// pixel of every stream.  Shared memory holds a run of slots as [16-byte piece of channels][slot]: that IS the tensor core's
// K-major layout without swizzle (eight rows of 16 bytes are a core matrix, row groups 128 bytes apart), whose start address
// may be any slot.  So an activation is staged once and every tap is another start address: no column buffer, no copy per
// tap, and rows of D that fall on zero slots are simply not stored.  Strided windows read one run of slots per parity of the
// source pixels; the input gradient of a strided layer runs as one class per parity of its pixels.
// A CTA stages, up to four warps issue the tile's products, all warps wait for them and store; two or three CTAs per SM overlap
// these phases.  Every wait is bounded and reports through the status word.
// (fp32 in this form, 3xTF32 with the split on the way into shared memory, was measured and left out: the accumulation truncates,
// so that the error of mma.sync's short chains is met only with a new accumulator every few k-steps, and with those 3 x 3 layers
// gain 1.1 to 1.4; pointwise ones have a kernel of their own, tl_conv_pw.cu.)
#include "tl_kernels.h"
#include "tl_tc.cuh"
#include <algorithm>

namespace tl {

int *tc_status_word();          // tl_conv_tc.cu

static constexpr int PX_MAXTAPS = 49, PX_THREADS = 256;

struct PxDiv { uint32_t m; int d; };            // n / d, exact while n d < 2^32
static PxDiv px_div(int d) { PxDiv r; r.d = d; r.m = d == 1 ? 0u : (uint32_t)(((1ull << 32) + d - 1) / d); return r; }
__device__ __forceinline__ PxDiv px_div_dev(int d) { PxDiv r; r.d = d; r.m = d == 1 ? 0u : 0xFFFFFFFFu / (uint32_t)d + 1u; return r; }
__device__ __forceinline__ int px_quot(int n, PxDiv d) { return d.m ? (int)__umulhi((uint32_t)n, d.m) : n; }

// Slots of a plane, and what the positions of a run are worked out with.
struct PxGeo {
    int n, Hp, Wp;                              // streams; rows and columns of slots
    int small, long_rows;                       // a run may span several planes / spans two rows at most
    PxDiv dWp, dplane, dHp;
};
// A tensor that runs of slots are staged from.
struct PxSrc {
    const __half *p;
    int C, H, W, S;                             // S: every S-th pixel, by parities
    int vec, nv; PxDiv dnv;                     // pixels of one load, loads of a row of slots
    int blocks, per;                            // warps that a run takes; channel groups of one of them at a time (px_deal)
    int nsub; unsigned char sub_r[9], sub_c[9]; // parities of the pixels that the taps read
};
struct PxClass { int Hc, Wc, oy0, ox0, tap0, ntaps, smin; };
struct PxFwd {
    PxGeo geo; PxSrc src;
    const __half *w, *bias; __half *dst; int *status;
    int Cd, oH, oW, osy, osx, KK;
    int wm, wk;                                 // weight index = m * wm + k * wk + tap
    PxClass cls[9];
    int at[PX_MAXTAPS];                         // a tap's start within the run, in 16-byte pieces
    unsigned char widx[PX_MAXTAPS];
    int tiles, MB, N, kg, groups, sl;           // 128-slot blocks of a tile; result channels; channels staged at a time, how often; slots of a run
    int tmem_cols, ksplit;                      // ksplit: issuers that share the taps of a block (one block: four, two: two)
    uint32_t b_off, raw_off, raw_bytes;         // bytes: weights, their copy in memory order (0: it passes through where the run will lie)
};
static __device__ __align__(16) uint32_t px_zeros[4];                      // what lanes outside the image read

__device__ __forceinline__ void px_sts(uint32_t to, uint32_t x0, uint32_t x1, uint32_t x2, uint32_t x3) { asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(to), "r"(x0), "r"(x1), "r"(x2), "r"(x3) : "memory"); }
__device__ __forceinline__ uint32_t px_lds16(uint32_t at) { unsigned short v; asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(at)); return v; }

// A run of sl slots from slot `base` of stream sta on, channels k0 .. k0 + 8 k8, by NW warps.  A lane takes V neighbouring
// pixels, works out once where they come from and where they go, and copies them for its share of the channels, eight at a
// time: eight loads of V pixels, V stores of eight channels.  Lanes outside the image read zeros from a fixed place instead of
// taking a branch.  lg = 0: [piece][slot][16 bytes].  lg = 1, 2, 3: [group of 2^lg pieces][slot][2^lg pieces], the pieces of a slot
// swizzled as the tensor core's layouts with rows of 32, 64 and 128 bytes want them; sl is a multiple of 32 then.  copies > 1 (of
// one group of pieces): the run again, one slot further each time, behind it.  ones >= 0: that channel, one past the last, is 1.
template <int V, int NW, int U> __device__ __forceinline__ void px_stage(const PxGeo &geo, const PxSrc &x, uint32_t to_sm, int lg, int sl, int copies, int ones, int k0, int k8, int base, int sta)
{
    const int lane = threadIdx.x & 31, Wp = geo.Wp, nv = x.nv, c_left = x.C - k0, plane = x.H * x.W;
    const __half *src = x.p + ((long long)sta * x.C + k0) * plane;
    const int row0 = geo.Hp > 1 ? px_quot(base, geo.dWp) : 0, er0 = (base - row0 * Wp) / V, gall = k8 * x.nsub, blocks = x.blocks, per = x.per;
    // the stores of a lane start at another pixel than its neighbours': eight lanes cover all banks
    const int rot = V == 4 ? (lane >> 1) & 3 : V == 2 ? (lane >> 2) & 1 : 0;
    int blk = threadIdx.x >> 5, part = 0;
    while (blk >= blocks) { blk -= blocks; part++; }
    while (part * per < gall) {
        const int er = er0 + blk * 32 + lane, dr = geo.long_rows ? (int)(er >= nv) : px_quot(er, x.dnv), j = er - dr * nv, row = row0 + dr;
        int st = 0, r = row;
        if (geo.Hp == 1) { st = row; r = 0; }
        else if (geo.small) { st = px_quot(row, geo.dHp); r = row - st * geo.Hp; }
        else if (row >= geo.Hp) { st = 1; r = row - geo.Hp; }
        const int s0 = row * Wp + j * V - base;                                         // slot of the first pixel
        const int i0 = max(0, -s0), i1 = min(V, min(Wp - j * V, sl - s0));              // pixels that are slots of the row and of the run
        const bool full = __all_sync(0xffffffffu, i0 == 0 && i1 == V);
        const bool in = i1 > i0 && (unsigned)(sta + st) < (unsigned)geo.n;
        const int g1 = min(gall, (part + 1) * per);
        for (int gr0 = part * per; gr0 < g1; gr0 += U) {
            uint32_t e[U][8][V == 4 ? 2 : 1], to[U]; int piece[U];
            const int pm = (1 << lg) - 1;
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int gr = min(gr0 + u, g1 - 1);
                int sp = 0, k = gr * 8, h = r, w = j * V;
                if (x.nsub > 1) { sp = gr / k8; k = (gr - sp * k8) * 8; }
                if (V == 1 && x.S > 1) { h = r * x.S + x.sub_r[sp]; w = w * x.S + x.sub_c[sp]; }
                const bool live = in && h < x.H && w < x.W;
                const __half *from = live ? src + (uint32_t)((st * x.C + k) * plane + h * x.W + w) : reinterpret_cast<const __half *>(px_zeros);
                const uint32_t step = live ? (uint32_t)plane : 0u;
                const int left = live ? c_left - k : 8;
#pragma unroll
                for (int q = 0; q < 8; q++) {
                    const __half *y = q < left ? from + q * step : reinterpret_cast<const __half *>(px_zeros);
                    if constexpr (V == 4) { const uint2 z = *reinterpret_cast<const uint2 *>(y); e[u][q][0] = z.x; e[u][q][1] = z.y; }
                    else if constexpr (V == 2) e[u][q][0] = *reinterpret_cast<const uint32_t *>(y);
                    else e[u][q][0] = *reinterpret_cast<const unsigned short *>(y);
                }
                if (ones >= 0 && k + 7 == ones) e[u][7][0] = e[u][7][V == 4 ? 1 : 0] = 0x3C003C00u;
                piece[u] = k / 8;
                to[u] = to_sm + (uint32_t)(sp * ((k8 + pm) >> lg) + (piece[u] >> lg)) * (uint32_t)(sl << (lg + 4));
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                if (gr0 + u >= g1) continue;
                if constexpr (V == 4) {
                    // rotate the four pixels by rot: words, then halves
#pragma unroll
                    for (int q = 0; q < 8; q++) {
                        const uint32_t a = rot & 2 ? e[u][q][1] : e[u][q][0], b = rot & 2 ? e[u][q][0] : e[u][q][1];
                        e[u][q][0] = __byte_perm(a, b, rot & 1 ? 0x5432 : 0x3210); e[u][q][1] = __byte_perm(a, b, rot & 1 ? 0x1076 : 0x7654);
                    }
                } else if constexpr (V == 2) {
#pragma unroll
                    for (int q = 0; q < 8; q++) e[u][q][0] = __byte_perm(e[u][q][0], 0, rot ? 0x1032 : 0x3210);
                }
#pragma unroll
                for (int i = 0; i < V; i++) {
                    const int pi = (i + rot) & (V - 1);
                    if (!(full || (pi >= i0 && pi < i1))) continue;
                    const uint32_t sel = i & 1 ? 0x7632 : 0x5410;
                    const uint32_t v0 = __byte_perm(e[u][0][i >> 1], e[u][1][i >> 1], sel), v1 = __byte_perm(e[u][2][i >> 1], e[u][3][i >> 1], sel);
                    const uint32_t v2 = __byte_perm(e[u][4][i >> 1], e[u][5][i >> 1], sel), v3 = __byte_perm(e[u][6][i >> 1], e[u][7][i >> 1], sel);
                    int s1 = s0 + pi;
                    uint32_t at = to[u];
                    for (int c = 0; c < copies && s1 >= 0; c++, s1--, at += (uint32_t)(sl << (lg + 4)))
                        px_sts(at + (uint32_t)((s1 << lg) | ((piece[u] ^ (s1 >> (3 - lg))) & pm)) * 16u, v0, v1, v2, v3);
                }
            }
        }
        blk += NW;
        while (blk >= blocks) { blk -= blocks; part++; }
    }
}
template <int NW, int U> __device__ __forceinline__ void px_run(const PxGeo &geo, const PxSrc &x, uint32_t to_sm, int lg, int sl, int copies, int ones, int k0, int k8, int base, int sta)
{
    if (x.vec == 4) px_stage<4, NW, U>(geo, x, to_sm, lg, sl, copies, ones, k0, k8, base, sta);
    else if (x.vec == 2) px_stage<2, NW, U>(geo, x, to_sm, lg, sl, copies, ones, k0, k8, base, sta);
    else px_stage<1, NW, U>(geo, x, to_sm, lg, sl, copies, ones, k0, k8, base, sta);
}

// The weights in memory have their taps innermost and every channel a stride apart, so that loads of single weights would touch a
// cache line per lane: contiguous pieces of them are copied to shared memory first and reordered from there, neighbouring lanes
// taking neighbouring taps, into [tap][piece][row][16 bytes].  A tap's weights start 16 bytes past a multiple of 128, so that
// those lanes store to different banks.
struct PxRows { int len, rows, rs, per, m_rows; };      // memory rows: one result channel (forward) or one source channel (input gradient) each
__device__ __forceinline__ PxRows px_rows(const PxFwd &p, int n0)
{
    PxRows r;
    const int live_n = min(p.N, p.Cd - n0);
    r.m_rows = p.wm > p.wk;
    r.len = r.m_rows ? p.src.C * p.KK : live_n * p.KK; r.rows = r.m_rows ? live_n : p.src.C; r.rs = r.m_rows ? p.wm : p.wk;
    r.per = min(r.rows, (int)(p.raw_bytes / (uint32_t)(r.len * 2)));
    if (!r.m_rows && r.per < r.rows) r.per &= ~7;
    return r;
}
__device__ __forceinline__ void px_fetch_weights(const PxFwd &p, const PxRows &r, uint32_t raw, int n0, int r0)
{
    const int tid = threadIdx.x, rn = min(r.per, r.rows - r0), total = rn * r.len;
    const __half *from = p.w + (long long)n0 * p.wm + (long long)r0 * r.rs;
    if ((r.rs == r.len || rn == 1) && (reinterpret_cast<uintptr_t>(from) & 15) == 0) {
        const int n16 = (total * 2 + 15) / 16;
        for (int e = tid; e < n16; e += PX_THREADS)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(raw + e * 16u), "l"(from + e * 8), "r"(min(16, total * 2 - e * 16)) : "memory");
    } else {
        const PxDiv dl = px_div_dev(r.len);
        constexpr int U = 8;
        for (int e0 = tid; e0 < total; e0 += U * PX_THREADS) {
            unsigned short v[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int e = e0 + u * PX_THREADS, row = px_quot(e, dl);
                v[u] = e < total ? *reinterpret_cast<const unsigned short *>(from + (long long)row * (r.rs - r.len) + e) : (unsigned short)0;
            }
#pragma unroll
            for (int u = 0; u < U; u++)
                if (e0 + u * PX_THREADS < total) asm volatile("st.shared.u16 [%0], %1;" ::"r"(raw + (uint32_t)(e0 + u * PX_THREADS) * 2u), "h"(v[u]) : "memory");
        }
    }
}
__device__ __forceinline__ void px_order_weights(const PxFwd &p, const PxRows &r, int ntaps, uint32_t raw, uint32_t b_sm, const int *tap_w, int n0, int r0)
{
    const int N = p.N, KK = p.KK, kpad = p.groups * p.kg, live_n = min(N, p.Cd - n0), rn = min(r.per, r.rows - r0);
    const bool last = r0 + rn >= r.rows;                                   // the last piece also fills the padding
    const int m_lo = r.m_rows ? r0 : 0, m_hi = r.m_rows && !last ? r0 + rn : N, k_lo = r.m_rows ? 0 : r0, k_hi = !r.m_rows && !last ? r0 + rn : kpad;
    const int mn = m_hi - m_lo, items = ntaps * mn * ((k_hi - k_lo) / 8);
    const PxDiv dt = px_div_dev(ntaps), dm = px_div_dev(mn);
    const uint32_t ks = (uint32_t)(r.m_rows ? KK : r.len) * 2u, ms = (uint32_t)(r.m_rows ? r.len : KK) * 2u, s_tap = (uint32_t)(kpad / 8 * N + 1) * 16u;
    constexpr int U = 2;
    for (int e0 = threadIdx.x; e0 < items; e0 += U * PX_THREADS) {
        uint32_t v[U][8], to[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int e = e0 + u * PX_THREADS, q1 = px_quot(e, dt), t = e - q1 * ntaps, q2 = px_quot(q1, dm), m = m_lo + q1 - q2 * mn, k = k_lo + q2 * 8;
            const int left = e < items && m < live_n ? p.src.C - k : 0;
            const uint32_t from = raw + (uint32_t)(m - m_lo) * ms + (uint32_t)(k - k_lo) * ks + (uint32_t)(e < items ? tap_w[t] : 0) * 2u;
            to[u] = b_sm + (uint32_t)t * s_tap + (uint32_t)((k / 8) * N + m) * 16u;
            if (left >= 8) {
#pragma unroll
                for (int q = 0; q < 8; q++) v[u][q] = px_lds16(from + q * ks);
            } else {
#pragma unroll
                for (int q = 0; q < 8; q++) v[u][q] = q < left ? px_lds16(from + q * ks) : 0u;
            }
        }
#pragma unroll
        for (int u = 0; u < U; u++)
            if (e0 + u * PX_THREADS < items) px_sts(to[u], v[u][0] | v[u][1] << 16, v[u][2] | v[u][3] << 16, v[u][4] | v[u][5] << 16, v[u][6] | v[u][7] << 16);
    }
}

// What bounds this kernel (128 streams of 24 -> 48 on 28 x 28): instructions around the tensor core, of which the products take a third
// (44 cycles each: both operands come from shared memory at 128 bytes a cycle); see the figures at the dispatch.
__global__ void __launch_bounds__(PX_THREADS, 3) conv_px_kernel(const __grid_constant__ PxFwd p)
{
    extern __shared__ __align__(1024) unsigned char px_smem[];
    __shared__ __align__(8) uint64_t bar;
    __shared__ uint32_t tmem_s;
    __shared__ int abort_s, tap_w[PX_MAXTAPS];
    __shared__ __align__(16) float bias_s[128];
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);      // (one value per warp, and known to be)
    const PxClass &c = p.cls[blockIdx.z];
    const int n0 = blockIdx.y * p.N, N = p.N, plane = p.geo.Hp * p.geo.Wp, ntaps = c.ntaps, smin = c.smin, sl = p.sl, MB = p.MB;
    const int k8_all = p.groups * p.kg / 8, k8 = p.kg / 8;                 // 16-byte pieces: of all channels, of a group
    const int issuers = min(MB * p.ksplit, 4);
    volatile int *abort_flag = &abort_s;
    // set-up that needs no data of the launches before this one
#pragma unroll
    for (int i = 0; i < (int)(sizeof(PxFwd) / 4); i += 16) asm volatile("" ::"r"(reinterpret_cast<const uint32_t *>(&p)[i]));
    if (warp == 0) { tc::tmem_alloc(&tmem_s, (uint32_t)p.tmem_cols); tc::tmem_relinquish(); }
    if (tid == 32) { tc::mbar_init(&bar, (uint32_t)issuers); tc::fence_barrier_init(); abort_s = 0; }
    if (tid >= 64 && tid < 64 + ntaps) tap_w[tid - 64] = p.widx[c.tap0 + tid - 64];
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tmem = tmem_s, a_sm = tc::smem_u32(px_smem), b_sm = a_sm + p.b_off;
    pdl_wait();

    const PxRows wr = px_rows(p, n0);
    const bool beside = p.raw_off != 0;                                    // the weights arrive while the first run of slots is staged
    if (ntaps) {
        if (beside) px_fetch_weights(p, wr, a_sm + p.raw_off, n0, 0);
        else
            for (int r0 = 0; r0 < wr.rows; r0 += wr.per) {
                px_fetch_weights(p, wr, a_sm, n0, r0);
                asm volatile("cp.async.wait_all;" ::: "memory");
                __syncthreads();
                px_order_weights(p, wr, ntaps, a_sm, b_sm, tap_w, n0, r0);
                __syncthreads();
            }
    }
    if (tid < N) bias_s[tid] = p.bias && n0 + tid < p.Cd ? __half2float(p.bias[n0 + tid]) : 0.f;

    const int cols_b = N * p.ksplit;                                       // accumulator columns of a block
    const long long dst_plane = (long long)p.oH * p.oW;
    uint32_t phase = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < p.tiles; tile += gridDim.x) {
        const int st0 = tile * (MB * 128) / plane, rem0 = tile * (MB * 128) - st0 * plane;
        int base = rem0 + smin, sta = st0;                                 // first slot of the run: at most one stream back
        if (base < 0) { base += plane; sta--; }
        for (int g = 0; g < p.groups; g++) {
            if (ntaps) {
                px_run<PX_THREADS / 32, 1>(p.geo, p.src, a_sm, 0, sl, 1, -1, g * p.kg, k8, base, sta);
                if (beside && tile == (int)blockIdx.x && g == 0) {
                    asm volatile("cp.async.wait_all;" ::: "memory");
                    __syncthreads();
                    px_order_weights(p, wr, ntaps, a_sm + p.raw_off, b_sm, tap_w, n0, 0);
                }
            }
            tc::fence_proxy_async();
            tc::tc_fence_before();
            if (__syncthreads_or(*abort_flag)) { ok = false; break; }
            if (ntaps == 0) continue;
            // ---- the products: up to four issuing warps (one thread starts a tcgen05 instruction every 120 to 180 cycles whatever its
            // size, several warps scale), each with blocks or, where a tile has fewer blocks than that, taps and accumulators of its
            // own.  A warp walks the loops together and elects a thread around the instructions: issued from a branch on one lane,
            // every operand takes a detour into uniform registers.
            if (warp < issuers) {
                tc::tc_fence_after();
                const uint64_t da = tc::smem_desc_kmajor(0u, (uint32_t)sl * 16u, 128u), db = tc::smem_desc_kmajor(0u, (uint32_t)N * 16u, 128u);
                const uint32_t a_hw = (uint32_t)(da >> 32), a_lw = (uint32_t)da + (a_sm >> 4), b_hw = (uint32_t)(db >> 32), b_lw = (uint32_t)db + (b_sm >> 4);
                const uint32_t idesc = tc::mma_idesc(tc::FMT_F16, 128, (uint32_t)N);
                const int b0 = warp % MB, t0 = p.ksplit > 1 ? warp / MB : 0;
                uint32_t more = g > 0;
                for (int t = t0; t < ntaps; t += p.ksplit) {
                    uint32_t aw = a_lw + (uint32_t)(p.at[c.tap0 + t] + b0 * 128), bw = b_lw + (uint32_t)((t * k8_all + g * k8) * N + t);
                    for (int ks = 0; ks < k8; ks += 2, aw += 2u * sl, bw += 2u * N) {
                        uint32_t d = tmem + (uint32_t)(b0 * cols_b + t0 * N), ab = aw;
                        for (int b = b0; b < MB; b += 4, ab += 512u, d += 4u * (uint32_t)cols_b)
                            if (tc::elect_one()) tc::mma_f16_ss(d, ((uint64_t)a_hw << 32) | ab, ((uint64_t)b_hw << 32) | bw, idesc, more);
                        more = 1u;
                    }
                }
                if (tc::elect_one()) tc::mma_commit(&bar);
                __syncwarp();
            }
            tc::wait_or_abort(&bar, phase, abort_flag, p.status, 51, 20u);
            phase ^= 1;
        }
        if (!ok) break;
        // ---- results: a thread holds 16 channels of one slot at a time, a warp stores 32 neighbouring pixels of a channel
        tc::tc_fence_after();
        const int ncg = N / 16, units = MB * ncg, nacc = min(p.ksplit, ntaps);
        __half *dst = p.dst + ((long long)st0 * p.Cd + n0) * dst_plane + (long long)c.oy0 * p.oW + c.ox0;
        int b = 0, cg = warp >> 2;
        while (cg >= ncg) { cg -= ncg; b++; }
        int bd = -1;
        long long at = 0; bool live = false;
        for (int u = warp >> 2; u < units; u += 2) {
            if (b != bd) {
                int x = rem0 + b * 128 + (warp & 3) * 32 + lane, st = 0;
                if (p.geo.small) { st = px_quot(x, p.geo.dplane); x -= st * plane; }
                else if (x >= plane) { st = 1; x -= plane; }
                const int r = p.geo.Hp > 1 ? px_quot(x, p.geo.dWp) : 0, cc = x - r * p.geo.Wp;
                live = st0 + st < p.geo.n && r < c.Hc && cc < c.Wc;
                at = (long long)st * p.Cd * dst_plane + (long long)(r * p.osy) * p.oW + cc * p.osx;
                bd = b;
            }
            float v[16];
            const uint32_t ta = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(b * cols_b + cg * 16);
            if (nacc) {
                tc::tmem_ld16w(ta, reinterpret_cast<uint32_t *>(v));
                tc::tmem_wait_ld();
                for (int s = 1; s < nacc; s++) {
                    uint32_t d[16];
                    tc::tmem_ld16w(ta + (uint32_t)(s * N), d);
                    tc::tmem_wait_ld();
#pragma unroll
                    for (int q = 0; q < 16; q++) v[q] += __uint_as_float(d[q]);
                }
            } else {
#pragma unroll
                for (int q = 0; q < 16; q++) v[q] = 0.f;
            }
            if (p.bias) {
                const float4 *bs = reinterpret_cast<const float4 *>(bias_s + cg * 16);
#pragma unroll
                for (int q = 0; q < 4; q++) { const float4 y = bs[q]; v[4 * q] += y.x; v[4 * q + 1] += y.y; v[4 * q + 2] += y.z; v[4 * q + 3] += y.w; }
            }
            if (live) {
                __half *o = dst + at + (long long)(cg * 16) * dst_plane;
                const int m_left = p.Cd - n0 - cg * 16;
                if (m_left >= 16) {
#pragma unroll
                    for (int q = 0; q < 16; q += 2) { const __half2 y = __floats2half2_rn(v[q], v[q + 1]); o[q * dst_plane] = __low2half(y); o[(q + 1) * dst_plane] = __high2half(y); }
                } else {
#pragma unroll
                    for (int q = 0; q < 16; q++) if (q < m_left) o[q * dst_plane] = __float2half_rn(v[q]);
                }
            }
            cg += 2;
            while (cg >= ncg) { cg -= ncg; b++; }
        }
        tc::tc_fence_before();
    }
    tc::tc_fence_before();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, (uint32_t)p.tmem_cols);
}

// ---------------------------------------------------------------- weight gradient
// dW[co][ci][t] = sum over slots of dY[slot][co] X[slot + shift_t][ci]: the same runs of slots, read MN-major (a core matrix is eight slots of
// eight channels either way), dY with zeros on the slots that are no pixel, so that the contraction runs over whole runs and a
// tap is again a start address.  Every tap has its accumulators in tensor memory, and so has, as a product with a column of ones, the
// bias gradient.  Twelve warps stage runs into two buffers while eight issue products, the taps dealt to them (a warp starts a
// product of these sizes every 200 cycles, ten of them one every 22).  Every CTA leaves one partial dW as [tap][four ci][co][ci] (neighbouring
// lanes of tensor memory are neighbouring co), which px_wg_reduce_kernel adds in CTA order.
// The tensor core truncates what it accumulates, so a chain of steps ends after about PXW_CHAIN of them: four more warps add its sums to a partial
// result, with ordinary rounding where they lie, sixteen bytes an instruction (four bytes an instruction made the kernel up to 1.8 times as
// slow).  The last chain is stored as a partial result of its own.  One chain for the life of a CTA (48 steps at 128 streams of
// 24 -> 48 on 28 x 28, 500 at 512 of 16 -> 39 on 48 x 48) left 0.4 and 3.5 % of the results beside the half nearest to the 64-bit value (mma.sync 0.1 %)
// and up to 9 % where all terms have one sign; so it is 0.2, 0.3 and 0.5 %, and the error against 64 bits that of the rounding to half
// precision to five digits.  Time before and after: 24.4 -> 24.9 us and 148 -> 129 there, 74 -> 78 at 300 of 64 -> 64 on 28 x 28, 191 -> 210 at 512
// of 7 -> 30, 5 x 5, on 48 x 47.
struct PxWg {
    PxGeo geo; PxSrc x, dy;
    float *part; int *status;
    int KK, tap0[4], ntaps[4];                  // taps of a slice of the grid (ntaps: products, of `copies` taps each)
    int at[PX_MAXTAPS];                         // a tap's start within the run of X, in 16-byte pieces
    int smin, ts, slx, sly, tiles, chains;      // slots of a tile; of a run of X, of dY; chains of a CTA
    int M, N, lgx, copies, ci_slices, tmem_cols, bias;  // lgx: rows of X are 2^lgx pieces
    long long group;                            // floats of one partial result
    uint32_t x_off, buf, ones_off;              // bytes: the run of X behind that of dY, the second pair of runs, 512 bytes of ones
};
static constexpr int PXW_STAGERS = 12, PXW_ISSUERS = 8, PXW_DRAINERS = 4, PXW_THREADS = 32 * (PXW_STAGERS + PXW_ISSUERS + PXW_DRAINERS), PXW_CHAIN = 32;

// Chains of about PXW_CHAIN steps, at most a quarter more: how many a CTA's steps make, and the step before which chain f of issuer i ends.
// The issuers end theirs in turn, spread over half a chain, so that the others keep the tensor cores busy.
static int px_wg_chains(int steps) { return steps <= PXW_CHAIN * 5 / 4 ? 1 : (steps + PXW_CHAIN - 1) / PXW_CHAIN; }
__device__ __forceinline__ int px_wg_chain_end(int f, int i, int issuers, int chains, int steps)
{
    const int turn = issuers > 1 ? 64 * i / (issuers - 1) : 32;                                    // 0 .. 64
    return f + 1 < chains ? (int)(((long long)steps * (128 * (f + 1) + turn - 32)) / (128 * chains)) : steps;
}
// Sixteen accumulators of a lane, neighbouring source channels, to the partial result, of which the first `left` exist: a CTA's first ones are
// stored, later ones added where they lie
__device__ __forceinline__ void px_wg_out(float *o, int step, int left, const uint32_t (&v)[16], bool first)
{
#pragma unroll
    for (int i = 0; i < 16; i += 4, o += step) {
        if (i >= left) break;
        if (first) asm volatile("st.global.v4.b32 [%0], {%1, %2, %3, %4};" ::"l"(o), "r"(v[i]), "r"(v[i + 1]), "r"(v[i + 2]), "r"(v[i + 3]) : "memory");
        else asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(o), "f"(__uint_as_float(v[i])), "f"(__uint_as_float(v[i + 1])),
                          "f"(__uint_as_float(v[i + 2])), "f"(__uint_as_float(v[i + 3])) : "memory");
    }
}

__global__ void __launch_bounds__(PXW_THREADS, 1) conv_px_wg_kernel(const __grid_constant__ PxWg p)
{
    extern __shared__ __align__(1024) unsigned char px_smem[];
    __shared__ __align__(8) uint64_t full[2], empty[2], done, chain_full[PXW_ISSUERS], chain_empty[PXW_ISSUERS];
    __shared__ uint32_t tmem_s;
    __shared__ int abort_s;
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);      // (one value per warp, and known to be)
    const int sl_t = blockIdx.y / p.ci_slices, ci0 = (blockIdx.y - sl_t * p.ci_slices) * p.N, ntaps = p.ntaps[sl_t], tap0 = p.tap0[sl_t];
    const int N = p.N, M = p.M, slx = p.slx, sly = p.sly, ts = p.ts, plane = p.geo.Hp * p.geo.Wp, k8x = N / 8, k8y = (p.dy.C + 7) / 8;
    const int copies = p.copies, NC = N * copies;                          // columns of a product
    // the bias gradient: a channel of ones where X has one to spare, else a product of its own
    const bool bias = p.bias && blockIdx.y == 0, fold = bias && ci0 + N > p.x.C;
    const int issuers = min(ntaps + (bias && !fold ? 1 : 0), PXW_ISSUERS); // (that product is dealt like one more tap)
    volatile int *abort_flag = &abort_s;
#pragma unroll
    for (int i = 0; i < (int)(sizeof(PxWg) / 4); i += 16) asm volatile("" ::"r"(reinterpret_cast<const uint32_t *>(&p)[i]));
    if (warp == PXW_STAGERS) { tc::tmem_alloc(&tmem_s, (uint32_t)p.tmem_cols); tc::tmem_relinquish(); }
    if (tid == 32) {
        for (int b = 0; b < 2; b++) { tc::mbar_init(&full[b], PXW_STAGERS); tc::mbar_init(&empty[b], (uint32_t)issuers); }
        tc::mbar_init(&done, (uint32_t)issuers);
        tc::fence_barrier_init();
        abort_s = 0;
    }
    if (tid >= 96 && tid < 96 + PXW_ISSUERS) { tc::mbar_init(&chain_full[tid - 96], 1); tc::mbar_init(&chain_empty[tid - 96], PXW_DRAINERS); tc::fence_barrier_init(); }
    const uint32_t base_sm = tc::smem_u32(px_smem), ones = base_sm + p.ones_off;
    if (tid >= 64 && tid < 96) px_sts(ones + (uint32_t)(tid - 64) * 16u, 0x3C003C00u, 0x3C003C00u, 0x3C003C00u, 0x3C003C00u);
    tc::fence_proxy_async();
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tmem = tmem_s;
    pdl_wait();

    const int t_begin = (int)((long long)p.tiles * blockIdx.x / gridDim.x), t_end = (int)((long long)p.tiles * (blockIdx.x + 1) / gridDim.x);
    const int steps = (t_end - t_begin) * (ts / 16), chains = p.chains, ncg = N / 16, bias_issuer = fold ? 0 : ntaps % issuers;
    // M = 64: sixteen rows in the first lanes of every quarter of tensor memory
    const int q = warp & 3, co = M == 64 ? q * 16 + lane : q * 32 + lane;
    const bool live = co < p.dy.C && (M == 128 || lane < 16);
    const uint32_t tq = tmem + ((uint32_t)(q * 32) << 16);
    const int c4 = (p.x.C + 3) / 4;
    // the last chain has a partial result of its own: added to the others' it would be waited for
    float *out = p.part + (long long)(blockIdx.x + (chains > 1 && warp < PXW_STAGERS ? gridDim.x : 0u)) * p.group, *out_bias = out + (long long)p.KK * c4 * p.dy.C * 4 + co;
    // taps t .. t_last of the slice from column group cg on (sixteen columns: source channels), every by-th group
    auto drain = [&](int t, int cg, int t_last, int by, bool first) {
        const int step = p.dy.C * 4;
        while (cg >= ncg) { cg -= ncg; t++; }
        while (t <= t_last) {
            uint32_t v[16];
            tc::tmem_ld16w(tq + (uint32_t)((t * ncg + cg) * 16), v);
            float *o = out + (long long)((tap0 + t) * c4 + ci0 / 4 + cg * 4) * step + co * 4;
            tc::tmem_wait_ld();
            if (live) px_wg_out(o, step, p.x.C - ci0 - cg * 16, v, first);
            cg += by;
            while (cg >= ncg) { cg -= ncg; t++; }
        }
    };
    auto drain_bias = [&](bool first) {
        uint32_t v[16];
        tc::tmem_ld16w(tq + (uint32_t)(fold ? N - 16 : ntaps * NC), v);
        tc::tmem_wait_ld();
        if (live) { if (first) *out_bias = __uint_as_float(v[15]); else atomicAdd(out_bias, __uint_as_float(v[15])); }
    };
    if (warp < PXW_STAGERS) {
        for (int tile = t_begin, it = 0; tile < t_end; tile++, it++) {
            const uint32_t buf = base_sm + (it & 1 ? p.buf : 0u);
            if (it >= 2 && !tc::warp_wait_or_abort(&empty[it & 1], (uint32_t)((it >> 1) - 1) & 1u, abort_flag, p.status, 52, 20u, lane)) break;
            const int st0 = tile * ts / plane, rem0 = tile * ts - st0 * plane;
            int base = rem0 + p.smin, sta = st0;
            if (base < 0) { base += plane; sta--; }
            px_run<PXW_STAGERS, 2>(p.geo, p.x, buf + p.x_off, p.lgx, slx, p.copies, fold ? N - 1 : -1, ci0, k8x, base, sta);
            px_run<PXW_STAGERS, 2>(p.geo, p.dy, buf, 3, sly, 1, -1, 0, k8y, rem0, st0);
            tc::fence_proxy_async();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&full[it & 1]);
        }
    } else if (warp - PXW_STAGERS < issuers) {
        const int wi = warp - PXW_STAGERS;
        // MN-major: a row is a slot with 64, 32 or 16 channels, swizzled by its address, so that a run may start at any slot; eight
        // slots are 8 rows on (stride offset), the next channels a run of slots on (leading offset)
        const uint32_t rx = 16u << p.lgx;
        const uint64_t da = tc::smem_desc_swizzled(0u, (uint32_t)sly * 128u, 1024u, tc::LAYOUT_SW128);
        const uint64_t db = tc::smem_desc_swizzled(0u, (uint32_t)slx * rx, 8u * rx, p.lgx == 3 ? tc::LAYOUT_SW128 : p.lgx == 2 ? tc::LAYOUT_SW64 : tc::LAYOUT_SW32);
        const uint64_t d1 = tc::smem_desc_kmajor(ones, 128u, 256u);
        const uint32_t a_hw = (uint32_t)(da >> 32), b_hw = (uint32_t)(db >> 32);
        const uint32_t idesc = tc::mma_idesc(tc::FMT_F16, (uint32_t)M, (uint32_t)NC) | tc::IDESC_A_MN_MAJOR | tc::IDESC_B_MN_MAJOR;
        const uint32_t idesc1 = tc::mma_idesc(tc::FMT_F16, (uint32_t)M, 16u) | tc::IDESC_A_MN_MAJOR | tc::IDESC_B_MN_MAJOR;
        bool ok = true;
        int step = 0, chain = 0, chain_end = px_wg_chain_end(0, wi, issuers, chains, steps);
        uint32_t more = 0;
        for (int tile = t_begin, it = 0; ok && tile < t_end; tile++, it++) {
            const uint32_t buf = (base_sm + (it & 1 ? p.buf : 0u)) >> 4;
            if (!tc::warp_wait_or_abort(&full[it & 1], (uint32_t)(it >> 1) & 1u, abort_flag, p.status, 53, 20u, lane)) { ok = false; break; }
            tc::tc_fence_after();
            uint32_t aw = (uint32_t)da + buf;
            const uint32_t bw0 = (uint32_t)db + buf + (p.x_off >> 4);
            for (int k = 0; k < ts; k += 16, aw += 128u, step++, more = 1u) {
                if (step == chain_end) {                                   // its sums are read before the next chain starts from zero
                    if (tc::elect_one()) tc::mma_commit(&chain_full[wi]);
                    __syncwarp();
                    if (!tc::warp_wait_or_abort(&chain_empty[wi], (uint32_t)chain & 1u, abort_flag, p.status, 63, 20u, lane)) { ok = false; break; }
                    tc::tc_fence_after();
                    chain_end = px_wg_chain_end(++chain, wi, issuers, chains, steps);
                    more = 0u;
                }
                const uint64_t ad = ((uint64_t)a_hw << 32) | aw;
                for (int t = wi; t < ntaps; t += issuers)
                    if (tc::elect_one()) tc::mma_f16_ss(tmem + (uint32_t)(t * NC), ad, ((uint64_t)b_hw << 32) | (bw0 + (uint32_t)(p.at[tap0 + t * copies] + (k << p.lgx))), idesc, more);
                if (bias && !fold && wi == bias_issuer && tc::elect_one()) tc::mma_f16_ss(tmem + (uint32_t)(ntaps * NC), ad, d1, idesc1, more);
                __syncwarp();
            }
            if (!ok) break;
            if (tc::elect_one()) tc::mma_commit(&empty[it & 1]);
            __syncwarp();
        }
        if (ok && tc::elect_one()) tc::mma_commit(&done);
        __syncwarp();
    } else if (warp >= PXW_STAGERS + PXW_ISSUERS) {
        // ---- all chains but the last, in the order in which they end
        bool ok = true;
        for (int f = 0; ok && f + 1 < chains; f++)
            for (int i = 0; i < issuers; i++) {
                ok = tc::warp_wait_or_abort(&chain_full[i], (uint32_t)f & 1u, abort_flag, p.status, 64, 20u, lane);
                if (!ok) break;
                tc::tc_fence_after();
                for (int t = i; t < ntaps; t += issuers)
                    drain(t * copies, 0, (t + 1) * copies - 1, 1, f == 0);
                if (bias && i == bias_issuer) drain_bias(f == 0);
                tc::tc_fence_before();
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(&chain_empty[i]);
            }
    }
    if (warp < PXW_STAGERS) {                                              // the last chains: three warps per quarter of tensor memory
        if (t_begin < t_end && tc::warp_wait_or_abort(&done, 0u, abort_flag, p.status, 54, 20u, lane)) {
            tc::tc_fence_after();
            drain(0, warp >> 2, ntaps * copies - 1, PXW_STAGERS / 4, true);
            if (bias && warp < 4) drain_bias(true);
        }
        tc::tc_fence_before();
    }
    __syncthreads();
    if (warp == PXW_STAGERS) { tc::tc_fence_after(); tc::tmem_dealloc(tmem, (uint32_t)p.tmem_cols); }
}

// 32 neighbouring elements x SL slices of the partial results per CTA; the slices are added in order.
// The products above also multiply the zeros of dY with pixels of X (on slots that are no result) and dY with zeros of X (the padding), which an
// infinite or NaN factor makes NaN.  So a sum that is no finite number is formed again by the whole CTA, from the pairs of pixels that the
// operator has; it is the only case in which X and dY are read.
struct PxWgSum { const float *part; const __half *x, *dy; __half *dw, *db; long long group; int groups, n, Ci, H, W, Co, Ho, Wo, S, padU, padL, Wk, KK, total; };
template <int SL>
__global__ void __launch_bounds__(32 * SL) px_wg_reduce_kernel(const __grid_constant__ PxWgSum p)
{
    pdl_wait();
    __shared__ float sums[SL][32];
    __shared__ uint32_t again_s;
    const int lane = threadIdx.x & 31, sl = threadIdx.x >> 5, e = blockIdx.x * 32 + lane, c4 = (p.Ci + 3) / 4;
    float acc = 0.f;
    if (e < p.total) {
        const float *src = p.part + e;
#pragma unroll 8
        for (int g = sl; g < p.groups; g += SL) acc += __ldcg(src + (long long)g * p.group);
    }
    sums[sl][lane] = acc;
    __syncthreads();
    bool again = false;
    if (sl == 0) {
#pragma unroll
        for (int s = 1; s < SL; s++) acc += sums[s][lane];
        const int q = (e >> 2) / p.Co, co = (e >> 2) - q * p.Co, t = q / c4, ci = (q - t * c4) * 4 + (e & 3);
        if (e < p.total && q >= c4 * p.KK) p.db[e - c4 * p.KK * p.Co * 4] = __float2half_rn(acc);
        else if (e < p.total && ci < p.Ci) { p.dw[((long long)co * p.Ci + ci) * p.KK + t] = __float2half_rn(acc); again = !isfinite(acc); }
        const uint32_t mask = __ballot_sync(0xffffffffu, again);
        if (lane == 0) again_s = mask;
    }
    if (!__syncthreads_or(again)) return;
    for (uint32_t left = again_s; left; left &= left - 1) {
        const int el = blockIdx.x * 32 + __ffs(left) - 1, q = (el >> 2) / p.Co, co = (el >> 2) - q * p.Co, t = q / c4, ci = (q - t * c4) * 4 + (el & 3);
        const int dh = t / p.Wk - p.padU, dw = t % p.Wk - p.padL, P = p.Ho * p.Wo;
        acc = 0.f;
        for (int i = threadIdx.x; i < p.n * P && !isnan(acc); i += 32 * SL) {
            const int s = i / P, r = (i - s * P) / p.Wo, h = r * p.S + dh, w = (i - s * P - r * p.Wo) * p.S + dw;
            if ((unsigned)h < (unsigned)p.H && (unsigned)w < (unsigned)p.W)
                acc = fmaf(__half2float(p.x[((long long)s * p.Ci + ci) * p.H * p.W + (long long)h * p.W + w]), __half2float(p.dy[((long long)s * p.Co + co) * P + (i - s * P)]), acc);
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        __syncthreads();
        if (lane == 0) sums[sl][0] = acc;
        __syncthreads();
        if (threadIdx.x == 0) {
#pragma unroll
            for (int s = 1; s < SL; s++) acc += sums[s][0];
            p.dw[((long long)co * p.Ci + ci) * p.KK + t] = __float2half_rn(acc);
        }
    }
}

// ---------------------------------------------------------------- host side
static int px_floordiv(int a, int b) { return a >= 0 ? a / b : -((-a + b - 1) / b); }

// Slots: zero columns and rows as far as the taps (row, column offsets of the source pixel) reach past the image of H x W pixels, of which
// results of Hc x Wc pixels are computed.  A tap's distance in slots goes to shift, its parity of source pixels to sub.
static bool px_slots(PxGeo &geo, PxSrc &x, int Hc, int Wc, int ntap, const int (*tap_rc)[2], int *shift, unsigned char *sub)
{
    const int S = x.S, Hsub = ceil_div(x.H, S), Wsub = ceil_div(x.W, S);
    int qr0 = 0, qr1 = 0, qc0 = 0, qc1 = 0;
    x.nsub = 0;
    for (int t = 0; t < ntap; t++) {
        const int qr = px_floordiv(tap_rc[t][0], S), qc = px_floordiv(tap_rc[t][1], S), a = tap_rc[t][0] - qr * S, b = tap_rc[t][1] - qc * S;
        qr0 = std::min(qr0, qr); qr1 = std::max(qr1, qr); qc0 = std::min(qc0, qc); qc1 = std::max(qc1, qc);
        int s = 0;
        while (s < x.nsub && !(x.sub_r[s] == a && x.sub_c[s] == b)) s++;
        if (s == x.nsub) { if (s == 9) return false; x.sub_r[s] = (unsigned char)a; x.sub_c[s] = (unsigned char)b; x.nsub++; }
        sub[t] = (unsigned char)s;
    }
    if (x.nsub == 0) return false;
    const long long Hp = std::max(Hsub - qr0, Hc + qr1), Wp = std::max(Wsub - qc0, Wc + qc1);
    if (Hp * Wp >= (1ll << 28) || (Hp > 1 && Hp * Wp * Wp >= (1ll << 32))) return false;        // (range of the quotients by multiplication)
    geo.Hp = (int)Hp; geo.Wp = (int)Wp;
    geo.dplane = px_div(geo.Hp * geo.Wp); geo.dWp = px_div(geo.Wp); geo.dHp = px_div(geo.Hp);
    for (int t = 0; t < ntap; t++) shift[t] = px_floordiv(tap_rc[t][0], S) * geo.Wp + px_floordiv(tap_rc[t][1], S);
    return true;
}
// pixels of one load: rows of whole vectors, aligned
static void px_vectors(PxSrc &x, int Wp)
{
    x.vec = 1;
    for (int v = 4; v > 1 && x.vec == 1; v /= 2)
        if (x.S == 1 && x.W % v == 0 && ((uintptr_t)x.p) % (v * 2) == 0) x.vec = v;
    x.nv = ceil_div(Wp, x.vec); x.dnv = px_div(x.nv);
}

// How a run of sl slots is dealt to nw warps: blocks of 32 loads (the most that any position of the run needs), and where they are fewer than
// the warps, the channel groups of a block shared.
static void px_deal(PxSrc &x, const PxGeo &geo, int sl, int gall, int nw)
{
    const int loads = geo.Wp >= sl ? sl / x.vec + 4 : (ceil_div(sl - 1, geo.Wp) + 1) * x.nv;
    x.blocks = ceil_div(std::max(1, loads), 32);
    x.per = ceil_div(gall, std::max(1, std::min(gall, nw / x.blocks)));
}

// What fits: result channels in slices, slots of a tile and channels staged at a time by shared memory and tensor-memory columns, chosen by
// a small model of the cycles.  false = not covered, nothing launched.
static bool px_launch(PxFwd &p, int ncls, const int (*tap_rc)[2])
{
    if (p.status == nullptr) return false;
    int Hc = 1, Wc = 1, taps_max = 0, ntap = 0, span = 0, smin_max = 0;
    for (int i = 0; i < ncls; i++) { Hc = std::max(Hc, p.cls[i].Hc); Wc = std::max(Wc, p.cls[i].Wc); taps_max = std::max(taps_max, p.cls[i].ntaps); ntap += p.cls[i].ntaps; }
    int shift[PX_MAXTAPS]; unsigned char sub[PX_MAXTAPS];
    if (!px_slots(p.geo, p.src, Hc, Wc, ntap, tap_rc, shift, sub)) return false;
    px_vectors(p.src, p.geo.Wp);
    const int plane = p.geo.Hp * p.geo.Wp;
    for (int i = 0; i < ncls; i++) {
        PxClass &c = p.cls[i];
        int lo = 1 << 30, hi = -(1 << 30);
        for (int t = c.tap0; t < c.tap0 + c.ntaps; t++) { lo = std::min(lo, shift[t]); hi = std::max(hi, shift[t]); }
        if (!c.ntaps) lo = hi = 0;
        c.smin = lo; span = std::max(span, hi - lo); smin_max = std::max(smin_max, lo);
    }
    if (span > 2048 || smin_max > 2048) return false;
    const int kpad = ceil_div(p.src.C, 16) * 16, npad = ceil_div(p.Cd, 16) * 16;
    if ((long long)p.geo.n * plane >= (1ll << 31) - 65536) return false;        // slots are counted in 32 bits
    const long long blocks = ((long long)p.geo.n * plane + 127) / 128;
    double best = 1e30;
    PxFwd bp = p;
    int best_ctas = 1;
    for (int ns = ceil_div(npad, 128); ns <= std::min(npad / 16, ceil_div(npad, 128) + 4); ns++) {
        const int N = ceil_div(ceil_div(p.Cd, ns), 16) * 16;
        if (ceil_div(p.Cd, N) != ns || ns > 65535) continue;
        const size_t row_b = p.wm > p.wk ? (size_t)p.src.C * p.KK * 2 : (size_t)8 * N * p.KK * 2, raw_b = ((size_t)std::min(N, p.Cd) * p.src.C * p.KK * 2 + 15) & ~(size_t)15;
        for (int ctas = 3; ctas >= 1; ctas--) {
            const size_t limit = (size_t)(ctas == 3 ? 74 : ctas == 2 ? 112 : 222) * 1024;
            for (int parts = 1; parts <= kpad / 16; parts *= 2) {
                const int kg = ceil_div(ceil_div(kpad, parts), 16) * 16, groups = ceil_div(kpad, kg);
                const size_t wb = (size_t)taps_max * ((size_t)groups * kg * N * 2 + 16);
                if (wb >= limit) continue;
                for (int MB = 8; MB >= 1; MB--) {
                    const int ksplit = taps_max > 1 ? (MB == 1 ? 4 : MB == 2 ? 2 : 1) : 1, cols_need = MB * N * ksplit;
                    int cols = 32;
                    while (cols < cols_need) cols *= 2;
                    if (cols * ctas > 512) continue;
                    const int sl = (MB * 128 + span) | 1;                  // odd: the pieces of a slot lie in different banks
                    const size_t ab = ((size_t)p.src.nsub * kg * 2 * sl + 127) & ~(size_t)127;
                    if (ab + wb > limit || ab < row_b) continue;
                    if ((double)(sl / plane + 3) * p.src.C * p.src.H * p.src.W >= 2147483648.0) continue;      // offsets within a run are 32 bits of elements
                    const long long tiles = (blocks + MB - 1) / MB;
                    if (tiles >= (1 << 30)) continue;
                    // cycles of a CTA: per tile staging, products and stores, which the CTAs of an SM share, and what does not shrink with it
                    const double stage = (double)p.src.nsub * kpad / 8 * sl * (p.src.vec == 4 ? 0.35 : p.src.vec == 2 ? 0.5 : 0.8), mma = (double)MB * taps_max * (kpad / 16) * std::max(50.0, N / 2.0);
                    const double epi = (double)MB * N * 4 * 4.0, fixed = 2000.0 + 900.0 * groups, wload = (double)taps_max * kpad / 8 * N * 0.3 + 1500.0;
                    const long long per_sm = (tiles * ns * ncls + sm_count() - 1) / sm_count();        // tiles of the busiest SM
                    const int live = (int)std::min<long long>(ctas, per_sm);
                    const double busy = per_sm * (stage + mma + epi), serial = (double)((per_sm + live - 1) / live) * (fixed + stage + mma + epi);
                    const double cost = std::max(busy, serial) + live * wload;
                    if (cost >= best) continue;
                    best = cost; best_ctas = ctas;
                    bp = p;
                    bp.MB = MB; bp.N = N; bp.kg = kg; bp.groups = groups; bp.sl = sl; bp.ksplit = ksplit; bp.tmem_cols = cols; bp.tiles = (int)tiles;
                    for (int i = 0; i < ncls; i++)
                        for (int t = p.cls[i].tap0; t < p.cls[i].tap0 + p.cls[i].ntaps; t++) bp.at[t] = sub[t] * (kg / 8) * sl + shift[t] - p.cls[i].smin;
                    bp.b_off = (uint32_t)ab;
                    px_deal(bp.src, p.geo, sl, kg / 8 * p.src.nsub, PX_THREADS / 32);
                    bp.geo.small = plane < sl + smin_max; bp.geo.long_rows = p.geo.Wp >= sl + 8;
                    bp.raw_off = ab + wb + raw_b <= limit ? (uint32_t)(ab + wb) : 0u;
                    bp.raw_bytes = bp.raw_off ? (uint32_t)raw_b : bp.b_off;
                }
            }
        }
    }
    if (best >= 1e30) return false;
    const int ns = ceil_div(p.Cd, bp.N);
    const size_t smem = bp.raw_off ? bp.raw_off + bp.raw_bytes : bp.b_off + (size_t)taps_max * ((size_t)bp.groups * bp.kg * 2 * bp.N + 16);
    static bool attr = false;
    if (!attr) { cudaFuncSetAttribute(conv_px_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 224 * 1024); attr = true; }
    const int gx = std::min(bp.tiles, std::max(1, sm_count() * best_ctas / (ns * ncls)));
    TL_LAUNCH(conv_px_kernel, dim3(gx, ns, ncls), PX_THREADS, smem, bp);
    return true;
}

// A pointwise layer of stride 1 is a product over the flattened plane: no slot is empty.
static ConvGeom px_flat(ConvGeom g)
{
    if (g.Hk == 1 && g.Wk == 1 && g.sh == 1 && g.sw == 1 && g.padU == 0 && g.padL == 0 && g.Hin == g.Hout && g.Win == g.Wout) { g.Win *= g.Hin; g.Wout = g.Win; g.Hin = g.Hout = 1; }
    return g;
}
static bool px_covers(const ConvGeom &g)
{
    return !g.depthwise && gemm_path() == 0 && g.Hk * g.Wk <= PX_MAXTAPS && g.sh == g.sw && g.sh <= 3 && g.padU <= 100 && g.padL <= 100 &&
           (long long)g.Hin * g.Win < (1ll << 28) && (long long)g.Hout * g.Wout < (1ll << 28);
}
// Where these kernels pay: their set-up (barriers, tensor memory, the reordered weights, the wait for the products) is 3 to 4 us more than
// that of the mma.sync kernels, their time per multiply-add half to a third.  Measured over ninety random layers (us, mma.sync /
// here, work in million multiply-adds with channels padded to 16):
//   forward, stride 1: 128 streams of 24 -> 48 on 28 x 28 (1390) 27.8 / 15.3; 300 of 64 -> 64 on 28 x 28 (8670) 89.7 / 50.4; 131 of 2 -> 8 on
//     19 x 30 (172) 10.0 / 8.9; 10 of 2 -> 40 on 28 x 48 (93) 7.5 / 7.4; 67 of 1 -> 15 on 18 x 17 (47) 6.0 / 7.3; many source channels
//     want more: 25 of 54 -> 6 on 36 x 42 (348) 12.4 / 14.1, 356 of 41 -> 13 on 21 x 11 (568) 19.5 / 18.1
//   forward, stride 2 (one load a pixel): 54 of 43 -> 22 on 23 x 34 (152) 11.7 / 18.7; 335 of 3 -> 6 on 36 x 37 (264) 17.7 / 20.7; 321 of
//     7 -> 58 on 39 x 39 (1183) 32.2 / 24.4
//   input gradient, stride 2 (a class per parity): 51 of 14 -> 5 on 32 x 30 (28) 7.8 / 8.1; 54 of 43 -> 22 on 23 x 34 (152) 21.2 / 12.3
//   1 x 1 (stride 1: what the products of tl_gemm_tma.cu decline): 70 of 20 -> 70 on 19 x 21 (72) 18.8 / 8.0, on even planes, which
//     mma.sync stages two pixels at a time, 72 of 13 -> 126 on 26 x 22 (84) 1.4 us slower for the two directions; stride 2: 42 of 8 -> 59
//     on 39 x 42 (18) 6.8 / 6.2 and 12.3 / 11.0, 207 of 34 -> 55 on 10 x 23 (38) 11.8 / 7.5 and 18.7 / 9.9
static double px_work(const ConvGeom &g) { return (double)g.n * g.Hout * g.Wout * g.Hk * g.Wk * (ceil_div(g.Cin, 16) * 16) * (ceil_div(g.Cout, 16) * 16); }
static bool px_pays(const ConvGeom &g, bool ig)
{
    const double w = px_work(g);
    if (g.Hk * g.Wk == 1) return w >= (g.sh > 1 ? 1.5e7 : g.Hin * g.Win % 2 ? 5e7 : 1.5e8);
    if (g.sh == 1) return w >= ((ig ? g.Cout : g.Cin) > 32 ? (ig ? 5e8 : 4e8) : 1e8);
    return w >= (ig ? 6e7 : 1e9);
}
// The weight gradient, with the bias gradient (a kernel and its sum less where there is one): 128 of 24 -> 48 on 28 x 28 36.0 / 23.9; 30 of
// 40 -> 80, 5 x 5, on 41 x 41 182 / 45; 1 of 24 -> 45 on 39 x 27 (15) 11.5 / 9.9; 56 of 11 -> 8 on 8 x 15 (15) 8.4 / 10.1.  Sixteen result
// channels fill a quarter of the rows of a product: 3 x 3 layers stay (262 of 27 -> 11 on 27 x 35 34.8 / 39.8), larger windows do
// not (30 of 42 -> 6, 5 x 5, on 29 x 25 37.2 / 19.1).  1 x 1: only where the products of tl_gemm_tma.cu would have to pack odd planes
// (100 of 96 -> 96 on 15 x 17 21.6 / 15.9), and strided (207 of 34 -> 55 on 10 x 23 14.1 / 9.9).
static bool px_wg_pays(const ConvGeom &g)
{
    const double w = px_work(g);
    if (g.Hk * g.Wk == 1) return g.sh == 1 ? g.n >= 2 && g.Hin * g.Win >= 64 && (g.Hin * g.Win) % 8 != 0 && g.Cin >= 32 && g.Cout >= 32 && w >= 5e7 : w >= 3e7;
    if (g.Hk * g.Wk <= 9) return g.Cout > 16 && w >= (g.n == 1 ? 1.4e7 : 2.5e7);
    return w >= 2e6;
}

// false = not covered, nothing launched
bool conv_px_fw(const ConvGeom &geom, const __half *x, const __half *w, const __half *bias, __half *y)
{
    const ConvGeom g = px_flat(geom);
    if (!px_covers(g) || !px_pays(geom, false)) return false;
    PxFwd p = {};
    int rc[PX_MAXTAPS][2];
    p.src.p = x; p.w = w; p.bias = bias; p.dst = y; p.status = tc_status_word(); p.geo.n = g.n; p.src.C = g.Cin; p.src.H = g.Hin; p.src.W = g.Win; p.Cd = g.Cout; p.oH = g.Hout; p.oW = g.Wout;
    p.src.S = g.sh; p.osy = p.osx = 1; p.KK = g.Hk * g.Wk; p.wm = g.Cin * p.KK; p.wk = p.KK;
    for (int t = 0; t < p.KK; t++) { rc[t][0] = t / g.Wk - g.padU; rc[t][1] = t % g.Wk - g.padL; p.widx[t] = (unsigned char)t; }
    p.cls[0] = {g.Hout, g.Wout, 0, 0, 0, p.KK, 0};
    return px_launch(p, 1, rc);
}
bool conv_px_ig(const ConvGeom &geom, const __half *dy, const __half *w, __half *dx)
{
    const ConvGeom g = px_flat(geom);
    if (!px_covers(g) || !px_pays(geom, true)) return false;
    const int s = g.sh;
    PxFwd p = {};
    int rc[PX_MAXTAPS][2];
    p.src.p = dy; p.w = w; p.bias = nullptr; p.dst = dx; p.status = tc_status_word(); p.geo.n = g.n; p.src.C = g.Cout; p.src.H = g.Hout; p.src.W = g.Wout; p.Cd = g.Cin; p.oH = g.Hin; p.oW = g.Win;
    p.src.S = 1; p.osy = p.osx = s; p.KK = g.Hk * g.Wk; p.wm = p.KK; p.wk = g.Cin * p.KK;
    int tap = 0, ncls = 0;
    for (int ph = 0; ph < s; ph++)
        for (int pw = 0; pw < s; pw++) {
            if (ph >= g.Hin || pw >= g.Win) continue;
            PxClass &c = p.cls[ncls++];
            c = {(g.Hin - ph + s - 1) / s, (g.Win - pw + s - 1) / s, ph, pw, tap, 0, 0};
            const int rh = (ph + g.padU) % s, qh = (ph + g.padU) / s, rw = (pw + g.padL) % s, qw = (pw + g.padL) / s;
            for (int kh = rh; kh < g.Hk; kh += s)
                for (int kw = rw; kw < g.Wk; kw += s) { rc[tap][0] = qh - (kh - rh) / s; rc[tap][1] = qw - (kw - rw) / s; p.widx[tap] = (unsigned char)(kh * g.Wk + kw); tap++; }
            c.ntaps = tap - c.tap0;
        }
    return px_launch(p, ncls, rc);
}

// Weight gradient, and the bias gradient where db is given.  false = not covered, nothing launched.
bool conv_px_wg(Scope &sc, const ConvGeom &geom, const __half *x, const __half *dy, __half *dw, __half *db)
{
    const ConvGeom g = px_flat(geom);
    if (!px_covers(g) || !px_wg_pays(geom) || g.Cout > 128) return false;
    PxWg p = {};
    int rc[PX_MAXTAPS][2];
    p.KK = g.Hk * g.Wk; p.status = tc_status_word();
    if (!p.status) return false;
    p.geo.n = g.n;
    p.x.p = x; p.x.C = g.Cin; p.x.H = g.Hin; p.x.W = g.Win; p.x.S = g.sh;
    p.dy.p = dy; p.dy.C = g.Cout; p.dy.H = g.Hout; p.dy.W = g.Wout; p.dy.S = 1; p.dy.nsub = 1;
    for (int t = 0; t < p.KK; t++) { rc[t][0] = t / g.Wk - g.padU; rc[t][1] = t % g.Wk - g.padL; }
    int shift[PX_MAXTAPS]; unsigned char sub[PX_MAXTAPS];
    if (!px_slots(p.geo, p.x, g.Hout, g.Wout, p.KK, rc, shift, sub)) return false;
    px_vectors(p.x, p.geo.Wp); px_vectors(p.dy, p.geo.Wp);
    int lo = 1 << 30, hi = -(1 << 30);
    for (int t = 0; t < p.KK; t++) { lo = std::min(lo, shift[t]); hi = std::max(hi, shift[t]); }
    if (hi - lo > 1024 || lo > 1024) return false;
    p.smin = lo;
    const int plane = p.geo.Hp * p.geo.Wp, span = hi - lo, k8y = ceil_div(g.Cout, 8);
    p.M = g.Cout <= 64 ? 64 : 128; p.bias = db != nullptr;
    const long long slots = (long long)g.n * plane, nw = (long long)g.Cout * g.Cin * p.KK;
    if (nw >= (1ll << 30)) return false;
    if (slots >= (1ll << 31) - 65536) return false;                        // slots are counted in 32 bits
    double best = 1e30;
    PxWg bp = p;
    int bgx = 0, bslices = 0;
    size_t bsmem = 0;
    for (int cis = ceil_div(g.Cin, 256); cis <= std::min(ceil_div(g.Cin, 16), ceil_div(g.Cin, 256) + 7); cis++) {
        const int N = ceil_div(ceil_div(g.Cin, cis), 16) * 16;
        if (N > 256 || ceil_div(g.Cin, N) != cis || cis > 16383) continue;
        // taps of a filter row as one product: copies of the run one slot apart, where its channels are one row of a swizzled layout
        const int lgx = N % 64 == 0 ? 3 : N % 32 == 0 ? 2 : 1, copies = g.sh == 1 && N == 8 << lgx && N * g.Wk <= 256 ? g.Wk : 1, prods = p.KK / copies;
        const int tmax = (512 - 16) / (N * copies), tsl = tmax ? ceil_div(prods, tmax) : 5, per = ceil_div(prods, std::max(tsl, 1));
        if (tsl > 4) continue;
        const int slices = cis * tsl, gx_max = (int)std::max<long long>(1, std::min<long long>(sm_count() / slices, (32ll << 20) / nw));       // (partial results: 256 MB at most)
        for (int ts = 512; ts >= 64; ts -= 16) {
            const int slx = (ts + span + 31) & ~31, sly = (ts + 31) & ~31;
            const uint32_t yb = (uint32_t)ceil_div(k8y, 8) * sly * 128u, xb = (uint32_t)(p.x.nsub * ((N / 8) >> lgx) * copies) * slx * (16u << lgx), buf = yb + xb;
            // the products read M channels of dY whatever it has: rows past them are not used, but have to lie in shared memory
            const size_t over = (size_t)(p.M / 64) * sly * 128, end = buf + std::max<size_t>(buf, over), smem = ((end + 1023) & ~(size_t)1023) + 512;
            if (smem > 222 * 1024) continue;
            if ((double)(slx / plane + 3) * std::max((double)g.Cin * g.Hin * g.Win, (double)g.Cout * g.Hout * g.Wout) >= 2147483648.0) continue;      // offsets within a run
            const int tiles = (int)((slots + ts - 1) / ts), gx = std::min(gx_max, tiles), rounds = ceil_div(tiles, gx);
            const double mma = (double)ts / 16 * (per + (db && g.Cin % 16 == 0 ? 1 : 0)) * std::max(22.0, (p.M + N * copies) / 2.1), stage = ((double)p.x.nsub * N / 8 * slx * (p.x.vec == 4 ? 0.5 : p.x.vec == 2 ? 0.8 : 1.3) + (double)k8y * sly * (p.dy.vec == 4 ? 0.5 : p.dy.vec == 2 ? 0.8 : 1.3));
            const double cost = rounds * (std::max(mma, stage) + 500) + std::min(mma, stage) + (double)gx * p.KK * g.Cin * g.Cout / 4000.0;
            if (cost >= best) continue;
            best = cost; bp = p; bgx = gx; bslices = slices; bsmem = smem;
            bp.N = N; bp.lgx = lgx; bp.copies = copies; bp.ci_slices = cis; bp.ts = ts; bp.slx = slx; bp.sly = sly; bp.tiles = tiles;
            for (int i = 0; i < tsl; i++) { bp.tap0[i] = i * per * copies; bp.ntaps[i] = std::min(per, prods - i * per); }
            for (int t = 0; t < p.KK; t++) bp.at[t] = (sub[t] * ((N / 8) >> lgx) * slx + shift[t] - lo) << lgx;
            int cols = 32;
            while (cols < per * N * copies + 16) cols *= 2;
            bp.tmem_cols = cols;
            bp.x_off = yb; bp.buf = buf; bp.ones_off = (uint32_t)(smem - 512);
            px_deal(bp.x, p.geo, slx, N / 8 * p.x.nsub, PXW_STAGERS); px_deal(bp.dy, p.geo, sly, k8y, PXW_STAGERS);
            bp.geo.small = plane < slx + std::max(0, lo); bp.geo.long_rows = p.geo.Wp >= slx + 8;
        }
    }
    if (best >= 1e30) return false;
    bp.chains = px_wg_chains(ceil_div(bp.tiles, bgx) * (bp.ts / 16));
    const int total = p.KK * ceil_div(g.Cin, 4) * 4 * g.Cout + (db ? g.Cout : 0);
    bp.group = ceil_div(total, 4) * 4;
    const int groups = bp.chains > 1 ? 2 * bgx : bgx;
    bp.part = sc.try_scratch<float>((size_t)groups * bp.group);
    if (!bp.part) return false;
    static bool attr = false;
    if (!attr) { cudaFuncSetAttribute(conv_px_wg_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 224 * 1024); attr = true; }
    TL_LAUNCH(conv_px_wg_kernel, dim3(bgx, bslices), PXW_THREADS, bsmem, bp);
    profile_add_flops(2.0 * g.n * g.Hout * g.Wout * nw);
    const PxWgSum r = {bp.part, x, dy, dw, db, bp.group, groups, g.n, g.Cin, g.Hin, g.Win, g.Cout, g.Hout, g.Wout, g.sh, g.padU, g.padL, g.Wk, p.KK, total};
    if (groups <= 160) TL_LAUNCH(px_wg_reduce_kernel<8>, ceil_div(total, 32), 256, 0, r);
    else TL_LAUNCH(px_wg_reduce_kernel<16>, ceil_div(total, 32), 512, 0, r);
    return true;
}

} // namespace tl

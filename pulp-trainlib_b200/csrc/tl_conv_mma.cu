// Convolutions of any shape on the warp-level tensor-core instructions: forward, input gradient and weight gradient for
// fp16 (mma.sync.m16n8k16, fp32 accumulation) and for the fp32 layers that the tcgen05 kernels decline (plane widths that
// are no multiple of four pixels, odd channel counts, 5 x 5 windows, single streams: 3xTF32 on mma.sync.m16n8k8).
// [ref: lib/sources/pulp_conv2d_fp32.c:85-113 (FW), :294-333 (WG), :504-549 (IG); naive kernels pulp_conv_naive_fp32.c:198-516]
//
// One idea serves the three: activations are staged in shared memory CHANNELS-LAST, [pixel][channel], zero outside the
// image.  A filter tap or a stride is then only another start address of a pixel's row of channels, so fragments are read
// in place for every tap (ldmatrix for fp16, 4-byte loads for fp32) and no column buffer exists anywhere.  The pitch of a
// pixel is an odd number of 16-byte units: eight neighbouring pixels never share a bank.
//
// Precision: the accumulator of mma.sync truncates when it adds (measured here: -2.3e-5 relative after 512 same-sign steps),
// so fp32 products run in short chains from zero (one filter tap of at most 16 k-steps, or 32 pixels of a weight gradient)
// whose sums are added to fp32 registers with ordinary rounding.
#include "tl_kernels.h"
#include "tl_tc.cuh"
#include <algorithm>

namespace tl {

static constexpr int CM_MAXTAPS = 49;
static constexpr int CM_SMEM_MAX = 220 * 1024;

// n / d, exact while n d < 2^32: the host checks it for the planes, patches are bounded by shared memory
struct CmDiv { uint32_t m; int d; };
// Streams of a tile on planes of P < tile pixels.  Offsets inside a tile are 32 bits wide (bytes of a source, elements of a result): a
// stream has less than 2^25 elements on either side (checked where the path is chosen), a tile less than 2^29.
static int cm_streams(int tile, int P, int n, long long stream_elements)
{
    return (int)std::max(1ll, std::min<long long>(std::min(tile / P, n), ((1ll << 29) - 1) / stream_elements));
}
static CmDiv cm_div(int d) { CmDiv r; r.d = d; r.m = d == 1 ? 0u : (uint32_t)(((1ull << 32) + d - 1) / d); return r; }
__device__ __forceinline__ CmDiv cm_div_dev(int d) { CmDiv r; r.d = d; r.m = d == 1 ? 0u : 0xFFFFFFFFu / (uint32_t)d + 1u; return r; }
__device__ __forceinline__ int cm_quot(int n, CmDiv d) { return d.m ? (int)__umulhi((uint32_t)n, d.m) : n; }

__device__ __forceinline__ void cm_ldsm(uint32_t (&r)[4], uint32_t addr) { asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr)); }
__device__ __forceinline__ void cm_ldsm_t(uint32_t (&r)[4], uint32_t addr) { asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr)); }
__device__ __forceinline__ void cm_hmma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void cm_tmma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t cm_lds32(uint32_t addr) { uint32_t v; asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr)); return v; }

// A patch of the source plane(s), channels-last: `streams` x rows x cols pixels of `chans` channels (a multiple of 8 fp16 / 4
// fp32; channels at or past c_left read as zero).  One item = one pixel x 16 bytes of channels: neighbouring threads take
// neighbouring pixels, so the per-channel loads are coalesced and the 16-byte store is conflict-free.  Addresses are a
// CTA-uniform base plus a 32-bit byte offset (cm_streams keeps a tile's span below 2 GB).  `warp`: this warp's place in the deal;
// a caller that stages two things at once counts the second one's warps from the other end, so that on small tiles both are loaded
// at the same time by different warps.
template <class T, int NT>
__device__ __forceinline__ void cm_stage(uint32_t sm, const T *src, int streams, int streams_left, int rows, int cols, CmDiv dcols,
                                         int row0, int col0, int H, int W, int chans, int c_left, uint32_t cstride, uint32_t sstride, uint32_t pitch, int warp)
{
    constexpr int SZ = (int)sizeof(T);
    const char *base = reinterpret_cast<const char *>(src);
    const int groups = chans >> 3, lane = threadIdx.x & 31;
    const uint32_t cs = cstride * SZ;
    // Blocks of 32 items and groups of eight channels, warp by warp (both uniform in a warp); all loads of an item are issued
    // before its first store.
    if ((W & 1) == 0 && ((cstride | sstride) & 1) == 0 && (reinterpret_cast<uintptr_t>(base) & (2 * SZ - 1)) == 0) {
        // even rows: an item is two neighbouring pixels from an even column (both inside the image or both outside), one load per
        // channel for the two
        const int w_even = col0 & ~1, half = (col0 + cols + 1 - w_even) >> 1, rc_n = rows * half, items = streams * rc_n;
        const CmDiv dhalf = cm_div_dev(half);
        const int blocks = (items + 31) >> 5;
        int g = 0, blk = warp;
        while (blk >= blocks) { blk -= blocks; g++; }
        for (; g < groups;) {
            const int p = blk * 32 + lane;
            int st = 0, rc = p;
            if (streams > 1) { st = p / rc_n; rc = p - st * rc_n; }
            const int r = rows > 1 ? cm_quot(rc, dhalf) : 0, w = w_even + 2 * (rc - r * half), h = row0 + r, c = w - col0;
            const bool in = p < items;
            const bool ok = in && st < streams_left && (unsigned)h < (unsigned)H && (unsigned)w < (unsigned)W;
            uint32_t off = ok ? ((uint32_t)st * sstride + (uint32_t)(h * W + w)) * SZ + (uint32_t)(g * 8) * cs : 0u;
            const int left = ok ? c_left - g * 8 : 0;
            const uint32_t to = sm + (uint32_t)((st * rows + r) * cols + c) * pitch + (uint32_t)g * (8u * SZ);
            if constexpr (sizeof(T) == 2) {
                uint32_t e[8], v0[4], v1[4];
#pragma unroll
                for (int q = 0; q < 8; q++, off += cs) e[q] = q < left ? *reinterpret_cast<const uint32_t *>(base + off) : 0u;
#pragma unroll
                for (int q = 0; q < 4; q++) { v0[q] = __byte_perm(e[2 * q], e[2 * q + 1], 0x5410); v1[q] = __byte_perm(e[2 * q], e[2 * q + 1], 0x7632); }
                if (in && c >= 0) asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(to), "r"(v0[0]), "r"(v0[1]), "r"(v0[2]), "r"(v0[3]) : "memory");
                if (in && c + 1 < cols) asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(to + pitch), "r"(v1[0]), "r"(v1[1]), "r"(v1[2]), "r"(v1[3]) : "memory");
            } else {
                float2 e[8];
#pragma unroll
                for (int q = 0; q < 8; q++, off += cs) e[q] = q < left ? *reinterpret_cast<const float2 *>(base + off) : make_float2(0.f, 0.f);
#pragma unroll
                for (int q = 0; q < 2; q++) {
                    if (in && c >= 0) asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(to + 16u * q), "f"(e[4 * q].x), "f"(e[4 * q + 1].x), "f"(e[4 * q + 2].x), "f"(e[4 * q + 3].x) : "memory");
                    if (in && c + 1 < cols) asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(to + pitch + 16u * q), "f"(e[4 * q].y), "f"(e[4 * q + 1].y), "f"(e[4 * q + 2].y), "f"(e[4 * q + 3].y) : "memory");
                }
            }
            blk += NT / 32;
            while (blk >= blocks) { blk -= blocks; g++; }
        }
        return;
    }
    const int rc_n = rows * cols, pix = streams * rc_n, blocks = (pix + 31) >> 5;
    int g = 0, blk = warp;
    while (blk >= blocks) { blk -= blocks; g++; }
    while (g < groups) {
        const int p = blk * 32 + lane;
        int st = 0, rc = p;
        if (streams > 1) { st = p / rc_n; rc = p - st * rc_n; }
        const int r = rows > 1 ? cm_quot(rc, dcols) : 0, c = rc - r * cols, h = row0 + r, w = col0 + c;
        const bool ok = p < pix && st < streams_left && (unsigned)h < (unsigned)H && (unsigned)w < (unsigned)W;
        uint32_t off = ok ? ((uint32_t)st * sstride + (uint32_t)(h * W + w)) * SZ + (uint32_t)(g * 8) * cs : 0u;
        const int left = ok ? c_left - g * 8 : 0;
        constexpr int R = 2 * SZ;                                          // 32-bit registers of an item
        uint32_t v[R];
        if constexpr (sizeof(T) == 2) {
            unsigned short e[8];
#pragma unroll
            for (int q = 0; q < 8; q++, off += cs) e[q] = q < left ? *reinterpret_cast<const unsigned short *>(base + off) : (unsigned short)0;
#pragma unroll
            for (int q = 0; q < 4; q++) v[q] = (uint32_t)e[2 * q] | ((uint32_t)e[2 * q + 1] << 16);
        } else {
#pragma unroll
            for (int q = 0; q < 8; q++, off += cs) v[q] = q < left ? *reinterpret_cast<const uint32_t *>(base + off) : 0u;
        }
        if (p < pix) {
#pragma unroll
            for (int q = 0; q < R / 4; q++)
                asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(sm + (uint32_t)p * pitch + (uint32_t)g * (8u * SZ) + 16u * q), "r"(v[4 * q]), "r"(v[4 * q + 1]), "r"(v[4 * q + 2]), "r"(v[4 * q + 3]) : "memory");
        }
        blk += NT / 32;
        while (blk >= blocks) { blk -= blocks; g++; }
    }
}

// The same patch by asynchronous 4-byte copies (fp32 only): nothing waits, the next tile's patch arrives while this one is
// multiplied.  The caller commits and waits.
template <int NT>
__device__ __forceinline__ void cm_stage_async(uint32_t sm, const float *src, int streams, int streams_left, int rows, int cols, CmDiv dcols,
                                               int row0, int col0, int H, int W, int chans, int c_left, uint32_t cstride, uint32_t sstride, uint32_t pitch, int warp)
{
    const char *base = reinterpret_cast<const char *>(src);
    const int groups = chans >> 3, lane = threadIdx.x & 31, rc_n = rows * cols, pix = streams * rc_n, blocks = (pix + 31) >> 5;
    const uint32_t cs = cstride * 4;
    int g = 0, blk = warp;
    while (blk >= blocks) { blk -= blocks; g++; }
    while (g < groups) {
        const int p = blk * 32 + lane;
        int st = 0, rc = p;
        if (streams > 1) { st = p / rc_n; rc = p - st * rc_n; }
        const int r = rows > 1 ? cm_quot(rc, dcols) : 0, c = rc - r * cols, h = row0 + r, w = col0 + c;
        const bool ok = st < streams_left && (unsigned)h < (unsigned)H && (unsigned)w < (unsigned)W;
        uint32_t off = ok ? ((uint32_t)st * sstride + (uint32_t)(h * W + w)) * 4u + (uint32_t)(g * 8) * cs : 0u;
        const int left = ok ? c_left - g * 8 : 0;
        const uint32_t to = sm + (uint32_t)p * pitch + (uint32_t)g * 32u;
        if (p < pix) {
#pragma unroll
            for (int q = 0; q < 8; q++, off += cs)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(to + 4u * q), "l"(base + (q < left ? off : 0u)), "r"(q < left ? 4 : 0) : "memory");
        }
        blk += NT / 32;
        while (blk >= blocks) { blk -= blocks; g++; }
    }
}

// ---------------------------------------------------------------- forward and input gradient
// dst[m][oy0 + i osy][ox0 + j osx] = sum over taps t and source channels k of src[k][i S + dr_t][j S + dc_t] W[m][k][t].
// Forward: S = the stride, one class.  Input gradient: a class per parity (oy0, ox0) of the input pixels (osy = osx = the
// stride, S = 1), whose taps are the ones that reach that parity; the weights are read with the channel roles swapped.
struct CmClass { int Hc, Wc, oy0, ox0, tap0, ntaps, dr_min, dc_min, cols, wide_cols; CmDiv dW, dcols; };
struct CmFwd {
    const void *src, *w, *bias; void *dst;
    int n, Cs, Hs, Ws, Cd, oH, oW, S, osy, osx, KK;
    int wm, wk;                              // weight index = m * wm + k * wk + tap
    int ncls; CmClass cls[9];
    signed char dr[CM_MAXTAPS], dc[CM_MAXTAPS]; unsigned char widx[CM_MAXTAPS];
    int st_tile;                             // streams per tile (planes smaller than a tile), else 1
    int CKS, groups, cblk, resident;         // channels staged at a time, how often, k-steps per chain; weights loaded once per CTA
    uint32_t pitch, wpitch, w_off, patch2;   // bytes: pixel, weight row; offset of the weights behind the patch; of the second patch (0: none)
    int rows_max, linear, pairs;
    int ksplit, kshare;                      // CTAs of a cluster that share the source channels, channels of each
};

// CTAs per SM.  What bounds these kernels is issue at few warps, so a third one helps where the registers allow it without loss: fp16
// tiles of 16 and 32 channels (400 streams of 8 -> 20 on 9 x 11: 12.4 -> 10.0 us a direction; 50 of 30 -> 13, 5 x 5: 19.5 -> 16.7).
// The 64-channel tiles lose the overlap of their fragment loads (88 -> 96 us), the fp32 ones up to 6 %.
template <class T, int WM> constexpr int cm_ctas() { return sizeof(T) == 2 && WM == 1 ? 3 : 2; }
template <class T, int MT, int WM, int WN, int WK, int BN, bool KS = false>
__global__ void __launch_bounds__(32 * WM * WN * WK, cm_ctas<T, WM>()) conv_mma_kernel(const __grid_constant__ CmFwd p)
{
    // a first read of a parameter misses the constant cache, one after the other where an index depends on another one: all lines at once
#pragma unroll
    for (int i = 0; i < (int)(sizeof(CmFwd) / 4); i += 16) asm volatile("" ::"r"(reinterpret_cast<const uint32_t *>(&p)[i]));
    constexpr int NT = 32 * WM * WN * WK, BM = 16 * MT * WM, TN = BN / WN, N8 = TN / 8;
    constexpr int CK = sizeof(T) == 2 ? 16 : 8, SZ = (int)sizeof(T);
    constexpr bool HALF = sizeof(T) == 2;
    extern __shared__ __align__(16) unsigned char cm_smem[];
    __shared__ int tap_off[CM_MAXTAPS], tap_of[CM_MAXTAPS + 1];
    const CmClass &c = p.cls[blockIdx.z];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wk = warp / (WM * WN), wmn = warp % (WM * WN), wm = wmn / WN, wn = wmn % WN;
    const int m0 = blockIdx.y * BM;
    const uint32_t patch = (uint32_t)__cvta_generic_to_shared(cm_smem), wsm = patch + p.w_off;
    const int P = c.Hc * c.Wc, ntaps = c.ntaps;
    // rows longer than a tile are cut into tiles of their own: a tile then stages its columns only
    const bool wide = c.Wc > BN;
    const int tiles_r = wide ? (c.Wc + BN - 1) / BN : 0;
    const int tiles_s = P < BN ? 1 : wide ? c.Hc * tiles_r : (P + BN - 1) / BN;      // tiles of one stream
    const int cols = wide ? c.wide_cols : c.cols;
    const int tiles = (P < BN ? (p.n + p.st_tile - 1) / p.st_tile : p.n * tiles_s);
    // KS: one cluster per tile, whose CTAs have a share of the source channels each
    int bx = blockIdx.x, gx = gridDim.x, rank = 0;
    if constexpr (KS) {
        asm("mov.u32 %0, %%clusterid.x;" : "=r"(bx));
        asm("mov.u32 %0, %%nclusterid.x;" : "=r"(gx));
        asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    }
    const int koff = KS ? rank * p.kshare : 0, Cs = KS ? min(p.kshare, p.Cs - koff) : p.Cs;
    if (bx >= tiles) { pdl_wait(); return; }

    // the tables come from the arguments alone: they are made before the wait for the kernel in front
    for (int t = tid; t < p.KK; t += NT) tap_of[t] = -1;
    __syncthreads();
    for (int t = tid; t < ntaps; t += NT) {
        tap_off[t] = ((p.dr[c.tap0 + t] - c.dr_min) * cols + (p.dc[c.tap0 + t] - c.dc_min)) * (int)p.pitch;
        tap_of[p.widx[c.tap0 + t]] = t;
    }
    __syncthreads();
    pdl_wait();

    // Weights of channels k0 .. k0 + kc as [tap][BM][wpitch].  A thread takes one (m, k) pair (fp16: two neighbouring k), walks
    // its taps, which are contiguous in memory, nine loads in flight, and stores each to its tap's matrix: one or two
    // instructions per weight.  (Dealing single weights to threads cost twenty: a third of the kernel's time.)
    auto load_weights = [&](int k0, int kc) {
        constexpr int V = HALF ? 2 : 1;
        const int kp = kc / V, items = kp * BM, KK = p.KK;
        const bool m_first = p.wm < p.wk;                                           // neighbouring threads take neighbouring memory
        const CmDiv dq = cm_div_dev(m_first ? BM : kp);
        const uint32_t s_tap = (uint32_t)BM * p.wpitch;
        const T *w = reinterpret_cast<const T *>(p.w);
        for (int e = tid; e < items; e += NT) {
            const int eq = cm_quot(e, dq), er = e - eq * dq.d, m = m_first ? er : eq, k = (m_first ? eq : er) * V;
            const bool ok0 = m0 + m < p.Cd && k0 + k < Cs, ok1 = ok0 && k0 + k + 1 < Cs;
            const T *src = ok0 ? w + (long long)(m0 + m) * p.wm + (long long)(koff + k0 + k) * p.wk : w;
            const uint32_t to = wsm + (uint32_t)m * p.wpitch + (uint32_t)(k * SZ);
            for (int t0 = 0; t0 < KK; t0 += 9) {
                if constexpr (HALF) {
                    unsigned short lo[9], hi[9];
#pragma unroll
                    for (int u = 0; u < 9; u++) {
                        const bool in = t0 + u < KK;
                        lo[u] = in && ok0 ? *reinterpret_cast<const unsigned short *>(src + t0 + u) : (unsigned short)0;
                        hi[u] = in && ok1 ? *reinterpret_cast<const unsigned short *>(src + p.wk + t0 + u) : (unsigned short)0;
                    }
#pragma unroll
                    for (int u = 0; u < 9; u++) {
                        const int t = t0 + u < KK ? tap_of[t0 + u] : -1;
                        if (t >= 0) asm volatile("st.shared.b32 [%0], %1;" ::"r"(to + (uint32_t)t * s_tap), "r"((uint32_t)lo[u] | ((uint32_t)hi[u] << 16)) : "memory");
                    }
                } else {
#pragma unroll
                    for (int u = 0; u < 9; u++) {
                        const int t = t0 + u < KK ? tap_of[t0 + u] : -1;
                        if (t >= 0) asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(to + (uint32_t)t * s_tap), "l"(ok0 ? src + t0 + u : src), "r"(ok0 ? 4 : 0) : "memory");
                    }
                }
            }
        }
    };                                                                             // (fp32: copies in flight, the caller waits)
    if (p.resident) load_weights(0, p.groups * p.CKS);

    const CmDiv dcols = wide ? cm_div_dev(cols) : c.dcols, dW = c.dW;
    const long long src_plane = (long long)p.Hs * p.Ws, dst_plane = (long long)p.oH * p.oW;

    struct Geo { int s0, p0, i0, col_t, live, rows; };
    const int st_n = P < BN ? p.st_tile : 1;
    auto geometry = [&](int tile) {
        Geo q;
        const int ts = tile % tiles_s, row_t = wide ? ts / tiles_r : 0;
        q.s0 = P < BN ? tile * p.st_tile : tile / tiles_s;
        q.col_t = wide ? (ts - row_t * tiles_r) * BN : 0;
        q.p0 = P < BN ? 0 : wide ? row_t * c.Wc + q.col_t : ts * BN;
        q.i0 = wide ? row_t : cm_quot(q.p0, dW);
        q.live = P < BN ? min(st_n, p.n - q.s0) * P : wide ? min(BN, c.Wc - q.col_t) : min(BN, P - q.p0);      // output pixels of the tile
        const int last = P < BN ? P - 1 : q.p0 + q.live - 1;
        q.rows = ((wide ? q.i0 : cm_quot(last, dW)) - q.i0) * p.S + p.rows_max;                                 // rows_max: rows that one output row needs
        return q;
    };
    auto stage = [&](const Geo &q, int g, uint32_t to, bool async) {
        const int k0 = g * p.CKS;
        const T *src = reinterpret_cast<const T *>(p.src) + ((long long)q.s0 * p.Cs + koff + k0) * src_plane;
        if constexpr (!HALF)
            if (async) {
                cm_stage_async<NT>(to, src, st_n, p.n - q.s0, q.rows, cols, dcols, q.i0 * p.S + c.dr_min, q.col_t * p.S + c.dc_min, p.Hs, p.Ws, p.CKS, Cs - k0,
                                   (uint32_t)src_plane, (uint32_t)(p.Cs * src_plane), p.pitch, NT / 32 - 1 - warp);
                return;
            }
        cm_stage<T, NT>(to, src, st_n, p.n - q.s0, q.rows, cols, dcols, q.i0 * p.S + c.dr_min, q.col_t * p.S + c.dc_min, p.Hs, p.Ws, p.CKS, Cs - k0,
                        (uint32_t)src_plane, (uint32_t)(p.Cs * src_plane), p.pitch, NT / 32 - 1 - warp);
    };
    // two patches (fp32, weights resident): the next tile's channels are on their way while this tile is multiplied
    const bool two = !HALF && p.patch2 != 0;
    uint32_t cur = 0;
    if (two) stage(geometry(bx), 0, patch, true);

    for (int tile = bx; tile < tiles; tile += gx) {
        const Geo geo = geometry(tile);
        const int s0 = geo.s0, p0 = geo.p0, i0 = geo.i0, col_t = geo.col_t, live = geo.live, rows = geo.rows;
        // start addresses (in the patch) of the pixels this lane supplies fragments for
        constexpr int NB = HALF ? N8 / 2 : N8;
        uint32_t pix[NB];
#pragma unroll
        for (int j = 0; j < NB; j++) {
            int q = wn * TN + (HALF ? j * 16 + (lane & 7) + ((lane >> 4) & 1) * 8 : j * 8 + (lane >> 2));
            if (q >= live) q = 0;
            int st = 0, pp = p0 + q;
            if (P < BN) { st = q / P; pp = q - st * P; }
            const int i = wide ? i0 : cm_quot(pp, dW), jj = pp - i * c.Wc - col_t;
            pix[j] = patch + (uint32_t)(((st * rows + (i - i0) * p.S) * cols + jj * p.S) * (int)p.pitch) + (HALF ? (uint32_t)((lane >> 3) & 1) * 16u : (uint32_t)(lane & 3) * 4u);
        }
        float acc[MT][N8][4];
#pragma unroll
        for (int i = 0; i < MT; i++)
#pragma unroll
            for (int j = 0; j < N8; j++)
#pragma unroll
                for (int q = 0; q < 4; q++) acc[i][j][q] = 0.f;

        for (int g = 0; g < p.groups; g++) {
            const int k0 = g * p.CKS;
            uint32_t poff = 0;
            if (two) {
                asm volatile("cp.async.wait_all;" ::: "memory");
                __syncthreads();                                                    // this patch has landed, the other one is free
                poff = cur; cur ^= p.patch2;
                if (g + 1 < p.groups) stage(geo, g + 1, patch + cur, true);
                else if (tile + gx < tiles) stage(geometry(tile + gx), 0, patch + cur, true);
            } else {
                __syncthreads();                                                    // the patch (and the weights) are free again
                if (!p.resident) load_weights(k0, p.CKS);
                stage(geo, g, patch, false);
                if constexpr (!HALF) asm volatile("cp.async.wait_all;" ::: "memory");       // the weights
                __syncthreads();
            }
            const uint32_t wg = wsm + (uint32_t)(p.resident ? k0 * SZ : 0);
            const int nck = p.CKS / CK, nblk = (nck + p.cblk - 1) / p.cblk;
            for (int u = wk; u < ntaps * nblk; u += WK) {
                const int t = nblk == 1 ? u : u / nblk, ck0 = nblk == 1 ? 0 : (u - t * nblk) * p.cblk, ck1 = min(nck, ck0 + p.cblk);
                const uint32_t toff = (uint32_t)tap_off[t] + poff;
                const uint32_t wrow = wg + (uint32_t)((t * BM + wm * 16 * MT) * (int)p.wpitch);
                if constexpr (HALF) {
                    const uint32_t wa = wrow + (uint32_t)((lane & 7) + ((lane >> 3) & 1) * 8) * p.wpitch + (uint32_t)(lane >> 4) * 16u;
                    for (int ck = ck0; ck < ck1; ck++) {
                        uint32_t a[MT][4], b[NB][4];
#pragma unroll
                        for (int i = 0; i < MT; i++) cm_ldsm(a[i], wa + (uint32_t)(i * 16) * p.wpitch + ck * 32u);
#pragma unroll
                        for (int j = 0; j < NB; j++) cm_ldsm(b[j], pix[j] + toff + ck * 32u);
#pragma unroll
                        for (int i = 0; i < MT; i++)
#pragma unroll
                            for (int j = 0; j < NB; j++) { cm_hmma(acc[i][2 * j], a[i], b[j][0], b[j][1]); cm_hmma(acc[i][2 * j + 1], a[i], b[j][2], b[j][3]); }
                    }
                } else {
                    const uint32_t wa = wrow + (uint32_t)(lane >> 2) * p.wpitch + (uint32_t)(lane & 3) * 4u;
                    float tmp[MT][N8][4];
#pragma unroll
                    for (int i = 0; i < MT; i++)
#pragma unroll
                        for (int j = 0; j < N8; j++)
#pragma unroll
                            for (int q = 0; q < 4; q++) tmp[i][j][q] = 0.f;
#pragma unroll 2
                    for (int ck = ck0; ck < ck1; ck++) {
                        uint32_t ah[MT][4], al[MT][4];
#pragma unroll
                        for (int i = 0; i < MT; i++)
#pragma unroll
                            for (int q = 0; q < 4; q++)                             // a0 (r, k), a1 (r + 8, k), a2 (r, k + 4), a3 (r + 8, k + 4)
                                tc::split_tf32_fast(__uint_as_float(cm_lds32(wa + (uint32_t)(i * 16 + (q & 1) * 8) * p.wpitch + ck * 32u + (q >> 1) * 16u)), ah[i][q], al[i][q]);
                        uint32_t bh[N8][2], bl[N8][2];
#pragma unroll
                        for (int j = 0; j < N8; j++)
#pragma unroll
                            for (int h = 0; h < 2; h++) tc::split_tf32_fast(__uint_as_float(cm_lds32(pix[j] + toff + ck * 32u + h * 16u)), bh[j][h], bl[j][h]);
                        // the three terms of a product go to one accumulator: neighbouring instructions take different ones
#pragma unroll
                        for (int term = 0; term < 3; term++)
#pragma unroll
                            for (int j = 0; j < N8; j++)
#pragma unroll
                                for (int i = 0; i < MT; i++) cm_tmma(tmp[i][j], term == 0 ? al[i] : ah[i], term == 1 ? bl[j][0] : bh[j][0], term == 1 ? bl[j][1] : bh[j][1]);
                    }
#pragma unroll
                    for (int i = 0; i < MT; i++)
#pragma unroll
                        for (int j = 0; j < N8; j++)
#pragma unroll
                            for (int q = 0; q < 4; q++) acc[i][j][q] += tmp[i][j][q];
                }
            }
        }
        if constexpr (WK > 1) {
            // the K shares of the warps meet in shared memory, added in warp order
            __syncthreads();
            float *red = reinterpret_cast<float *>(cm_smem);
            if (wk > 0) {
#pragma unroll
                for (int i = 0; i < MT; i++)
#pragma unroll
                    for (int j = 0; j < N8; j++)
#pragma unroll
                        for (int q = 0; q < 4; q++) red[((((wk - 1) * WM * WN + wmn) * MT + i) * N8 + j) * 128 + q * 32 + lane] = acc[i][j][q];
            }
            __syncthreads();
            if (wk == 0)
#pragma unroll
                for (int k = 1; k < WK; k++)
#pragma unroll
                    for (int i = 0; i < MT; i++)
#pragma unroll
                        for (int j = 0; j < N8; j++)
#pragma unroll
                            for (int q = 0; q < 4; q++) acc[i][j][q] += red[((((k - 1) * WM * WN + wmn) * MT + i) * N8 + j) * 128 + q * 32 + lane];
            if constexpr (KS) {
                // then those of the cluster (which has one tile only) in the memory of its first CTA, in rank order
                float *own = red + (WK - 1) * WM * WN * MT * N8 * 128;
                if (wk == 0)
#pragma unroll
                    for (int i = 0; i < MT; i++)
#pragma unroll
                        for (int j = 0; j < N8; j++)
#pragma unroll
                            for (int q = 0; q < 4; q++) own[((wmn * MT + i) * N8 + j) * 128 + q * 32 + lane] = acc[i][j][q];
                asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
                if (wk == 0 && rank == 0) {
                    const uint32_t at = (uint32_t)__cvta_generic_to_shared(own) + (uint32_t)(wmn * MT * N8 * 128 + lane) * 4u;
                    for (int r = 1; r < p.ksplit; r++) {
                        uint32_t there;
                        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"(at), "r"(r));
                        float v[MT * N8 * 4];
#pragma unroll
                        for (int q = 0; q < MT * N8 * 4; q++) asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v[q]) : "r"(there + 128u * q) : "memory");
#pragma unroll
                        for (int i = 0; i < MT; i++)
#pragma unroll
                            for (int j = 0; j < N8; j++)
#pragma unroll
                                for (int q = 0; q < 4; q++) acc[i][j][q] += v[(i * N8 + j) * 4 + q];
                    }
                }
                if (rank > 0) continue;
            }
            if (wk > 0) continue;
        }
        // results: a lane holds pixel pairs of two rows (output channels) per 16 x 8 fragment
        T *dst = reinterpret_cast<T *>(p.dst) + (long long)s0 * p.Cd * dst_plane + (long long)c.oy0 * p.oW + c.ox0;
        const T *bias = reinterpret_cast<const T *>(p.bias);
        float bv[MT][2];
        T *row[MT][2];
#pragma unroll
        for (int i = 0; i < MT; i++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int m = m0 + wm * 16 * MT + i * 16 + (lane >> 2) + h * 8;
                row[i][h] = m < p.Cd ? dst + m * dst_plane : nullptr;
                bv[i][h] = bias && m < p.Cd ? ld(bias + m) : 0.f;
            }
#pragma unroll
        for (int j = 0; j < N8; j++) {
            const int q0 = wn * TN + 8 * j + 2 * (lane & 3);
            if (q0 >= live) continue;
            int off[2];
            const bool second = q0 + 1 < live;
            if (p.linear && P >= BN) { off[0] = p0 + q0; off[1] = off[0] + 1; }          // the class is the whole plane, pixels in memory order
            else
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    int st = 0, pp = p0 + q0 + (second ? h : 0);
                    if (P < BN) { st = pp / P; pp -= st * P; }
                    const int i = cm_quot(pp, dW), jj = pp - i * c.Wc;
                    off[h] = st * p.Cd * (int)dst_plane + i * p.osy * p.oW + jj * p.osx;
                }
            // one store for two pixels: even planes and an aligned tensor (pairs), from an even pixel (a tile inside a long row may start odd)
            const bool pair = p.pairs && second && off[1] == off[0] + 1 && (off[0] & 1) == 0;
#pragma unroll
            for (int i = 0; i < MT; i++)
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    if (!row[i][h]) continue;
                    const float v0 = acc[i][j][2 * h] + bv[i][h], v1 = acc[i][j][2 * h + 1] + bv[i][h];
                    if (pair) {
                        if constexpr (HALF) *reinterpret_cast<__half2 *>(row[i][h] + off[0]) = __floats2half2_rn(v0, v1);
                        else *reinterpret_cast<float2 *>(row[i][h] + off[0]) = make_float2(v0, v1);
                    } else {
                        st(row[i][h] + off[0], v0);
                        if (second) st(row[i][h] + off[1], v1);
                    }
                }
        }
    }
    if constexpr (KS) asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");      // no CTA leaves while its sums are read
}

template <class T, int MT, int WM, int WN, int WK, int BN, bool KS = false> static bool conv_mma_launch(CmFwd &p, int cpad, bool dry)
{
    constexpr int CK = sizeof(T) == 2 ? 16 : 8, SZ = (int)sizeof(T), BM = 16 * MT * WM;
    // the largest patch over the classes: streams x rows x cols
    long long pix = 0; int taps = 0, tiles_max = 0; p.st_tile = 1;
    const int P0 = p.cls[0].Hc * p.cls[0].Wc;                              // class 0 has the most pixels
    if (P0 < BN) p.st_tile = cm_streams(BN, P0, p.n, std::max((long long)p.Cs * p.Hs * p.Ws, (long long)p.Cd * p.oH * p.oW));
    for (int i = 0; i < p.ncls; i++) {
        const CmClass &c = p.cls[i];
        const int P = c.Hc * c.Wc;
        const bool wide = c.Wc > BN;
        if (!(wide && p.linear) && (long long)P * c.Wc >= (1ll << 32)) return false;          // (range of the quotients by multiplication)
        p.cls[i].wide_cols = (BN - 1) * p.S + c.cols - (c.Wc - 1) * p.S;
        const int rows = (wide ? 0 : P < BN ? c.Hc - 1 : (BN + c.Wc - 2) / c.Wc) * p.S + p.rows_max;
        pix = std::max(pix, (long long)p.st_tile * rows * (wide ? p.cls[i].wide_cols : c.cols));
        taps = std::max(taps, c.ntaps);
        tiles_max = std::max(tiles_max, P < BN ? ceil_div(p.n, p.st_tile) : (int)std::min<long long>((long long)p.n * (wide ? (long long)c.Hc * ceil_div(c.Wc, BN) : ceil_div(P, BN)), 1 << 30));
    }
    const size_t red = WK > 1 ? (size_t)(KS ? WK : WK - 1) * WM * WN * MT * (BN / WN / 8) * 512 : 0;
    auto plan = [&](int cks, bool resident, size_t limit, bool two) {
        p.CKS = cks; p.groups = ceil_div(cpad, cks); p.resident = resident;
        p.pitch = (uint32_t)(cks * SZ + 16); p.wpitch = (uint32_t)((resident ? p.groups * cks : cks) * SZ + 16);
        const size_t pb = std::max<size_t>(((size_t)pix * p.pitch + 15) & ~(size_t)15, red);
        p.patch2 = two ? (uint32_t)pb : 0u; p.w_off = (uint32_t)(two ? 2 * pb : pb);
        return p.w_off + (size_t)taps * BM * p.wpitch <= limit;
    };
    // everything resident in half of an SM's shared memory if it fits (two CTAs overlap staging and arithmetic), else fewer
    // channels at a time, else all of it, else weights reloaded with every group of channels
    bool ok = false;
    for (size_t limit : {(size_t)110 * 1024, (size_t)CM_SMEM_MAX}) {
        if (sizeof(T) == 4 && WK == 1)                                     // (the K shares of WK > 1 meet where the patches lie)
            for (int parts = 1; !ok && parts <= cpad / CK; parts *= 2) ok = plan(ceil_div(ceil_div(cpad, parts), CK) * CK, true, limit, true);
        if (ok) break;
        for (int parts = 1; !ok && parts <= cpad / CK; parts *= 2) ok = plan(ceil_div(ceil_div(cpad, parts), CK) * CK, true, limit, false);
        if (ok) break;
        for (int parts = 1; !ok && parts <= cpad / CK; parts *= 2) ok = plan(ceil_div(ceil_div(cpad, parts), CK) * CK, false, limit, false);
        if (ok) break;
    }
    if (!ok) return false;
    if (dry) return true;
    const int nck = p.CKS / CK;
    p.cblk = std::min(nck, 16);
    while (WK > 1 && p.cblk > 1 && taps * ceil_div(nck, p.cblk) < 2 * WK) p.cblk = (p.cblk + 1) / 2;
    const size_t smem = p.w_off + (size_t)taps * BM * p.wpitch;
    auto kern = conv_mma_kernel<T, MT, WM, WN, WK, BN, KS>;
    static size_t attr = 0;
    if (smem > attr) { cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, CM_SMEM_MAX); attr = CM_SMEM_MAX; }
    const int co_tiles = ceil_div(p.Cd, BM);
    // every CTA slot taken: co-resident CTAs share an SM, so a last round that only some of them have costs less than idle slots
    const int gx = std::min(tiles_max, std::max(1, sm_count() * (cm_ctas<T, WM>() == 3 && smem <= 74 * 1024 ? 3 : smem <= 110 * 1024 ? 2 : 1) / (co_tiles * p.ncls)));
    if constexpr (KS) TL_LAUNCH_CLUSTER((conv_mma_kernel<T, MT, WM, WN, WK, BN, true>), dim3(tiles_max * p.ksplit, co_tiles, p.ncls), 32 * WM * WN * WK, smem, p.ksplit, p);
    else TL_LAUNCH((conv_mma_kernel<T, MT, WM, WN, WK, BN, KS>), dim3(gx, co_tiles, p.ncls), 32 * WM * WN * WK, smem, p);
    return true;
}

template <class T> static bool conv_mma_dispatch(CmFwd &p)
{
    constexpr int CK = sizeof(T) == 2 ? 16 : 8;
    const int cpad = ceil_div(p.Cs, CK) * CK;
    if ((long long)p.Cs * p.Hs * p.Ws >= (1ll << 25) || (long long)p.Cd * p.oH * p.oW >= (1ll << 25)) return false;      // cm_streams
    p.linear = p.ncls == 1 && p.osx == 1 && p.osy == 1;
    p.pairs = p.linear && (p.oW * p.oH) % 2 == 0 && ((uintptr_t)p.dst) % (2 * sizeof(T)) == 0;
    long long tiles = 0;                                                   // 128-pixel tiles
    for (int i = 0; i < p.ncls; i++) tiles += ((long long)p.n * p.cls[i].Hc * p.cls[i].Wc + 127) / 128;
    // Few tiles (single streams): 16 x 32 result tiles whose taps and channels are dealt to four warps each, so that a layer of
    // 32 channels on 32 x 32 pixels still occupies 64 CTAs; otherwise 128 pixels by 16, 32 or 64 channels.
    if (2 * tiles * ceil_div(p.Cd, p.Cd > 32 ? 64 : 32) < sm_count()) {
        // Long sums under few tiles run at the speed of one CTA's chain of taps and channels.  A cluster that shares the channels costs
        // about 1 us more and pays from 48 products of 16 (fp32: 8) channels a pixel, with three CTAs or more and two per SM at most:
        // one stream of 96 -> 96 on 9 x 13 with stride 2, fp32, 13.4 -> 6.8 us forward and 8.9 -> 7.1 back, 256 -> 256 on 8 x 8 25.8 -> 9.3,
        // 512 -> 500 on 4 x 4 with 1 x 1 windows, whose weights bound it, fp16, 15.8 -> 8.1; but 32 -> 16 on 32 x 32 (36) 6.0 -> 6.2 and
        // 64 -> 64 on 32 x 32 with two CTAs 8.6 -> 8.9.
        const int nck = cpad / CK;
        int ctas = 0, taps = 0;
        for (int i = 0; i < p.ncls; i++) {
            const int P = p.cls[i].Hc * p.cls[i].Wc;
            ctas += P < 32 ? ceil_div(p.n * P, 32) : p.n * ceil_div(P, 32);
            taps = std::max(taps, p.cls[i].ntaps);
        }
        ctas *= ceil_div(p.Cd, 16);
        const int most = std::min(std::min(8, nck), 2 * sm_count() / ctas);
        if (most >= 3 && (taps * nck >= 48 || (taps == 1 && nck >= 24))) {
            p.kshare = ceil_div(nck, most) * CK;
            p.ksplit = ceil_div(cpad, p.kshare);
            if (conv_mma_launch<T, 1, 1, 2, 4, 32, true>(p, p.kshare, false)) return true;
        }
        return conv_mma_launch<T, 1, 1, 2, 4, 32>(p, cpad, false);
    }
    if (p.Cd > 32) return conv_mma_launch<T, 2, 2, 4, 1, 128>(p, cpad, false) || conv_mma_launch<T, 1, 1, 8, 1, 128>(p, cpad, false);
    if (p.Cd > 16) return conv_mma_launch<T, 2, 1, 8, 1, 128>(p, cpad, false) || conv_mma_launch<T, 1, 1, 8, 1, 128>(p, cpad, false);
    return conv_mma_launch<T, 1, 1, 8, 1, 128>(p, cpad, false);
}

// A pointwise layer of stride 1 is a product over the flattened plane: one long row, so tiles stage no pixel twice.
static ConvGeom cm_flat(ConvGeom g)
{
    if (g.Hk == 1 && g.Wk == 1 && g.sh == 1 && g.sw == 1 && g.padU == 0 && g.padL == 0 && g.Hin == g.Hout && g.Win == g.Wout) { g.Win *= g.Hin; g.Wout = g.Win; g.Hin = g.Hout = 1; }
    return g;
}

// false = not covered, nothing launched
template <class T> bool conv_mma_fw(const ConvGeom &geom, const T *x, const T *w, const T *bias, T *y)
{
    const ConvGeom g = cm_flat(geom);
    const int KK = g.Hk * g.Wk;
    if (g.depthwise || gemm_path() == 1 || KK > CM_MAXTAPS || g.sh != g.sw || (long long)g.Hin * g.Win >= (1ll << 31)) return false;
    CmFwd p;
    p.src = x; p.w = w; p.bias = bias; p.dst = y; p.n = g.n; p.Cs = g.Cin; p.Hs = g.Hin; p.Ws = g.Win; p.Cd = g.Cout; p.oH = g.Hout; p.oW = g.Wout;
    p.S = g.sh; p.osy = p.osx = 1; p.KK = KK; p.wm = g.Cin * KK; p.wk = KK; p.ncls = 1;
    for (int t = 0; t < KK; t++) { p.dr[t] = (signed char)(t / g.Wk - g.padU); p.dc[t] = (signed char)(t % g.Wk - g.padL); p.widx[t] = (unsigned char)t; }
    if (g.padU > 100 || g.padL > 100) return false;
    CmClass &c = p.cls[0];
    c.Hc = g.Hout; c.Wc = g.Wout; c.oy0 = c.ox0 = 0; c.tap0 = 0; c.ntaps = KK; c.dr_min = -g.padU; c.dc_min = -g.padL;
    c.cols = (g.Wout - 1) * g.sw + g.Wk; c.dW = cm_div(g.Wout); c.dcols = cm_div(c.cols);
    p.rows_max = g.Hk;
    return conv_mma_dispatch<T>(p);
}
template <class T> bool conv_mma_ig(const ConvGeom &geom, const T *dy, const T *w, T *dx)
{
    const ConvGeom g = cm_flat(geom);
    const int KK = g.Hk * g.Wk, s = g.sh;
    if (g.depthwise || gemm_path() == 1 || KK > CM_MAXTAPS || g.sh != g.sw || s > 3 || g.padU > 100 || g.padL > 100) return false;
    CmFwd p;
    p.src = dy; p.w = w; p.bias = nullptr; p.dst = dx; p.n = g.n; p.Cs = g.Cout; p.Hs = g.Hout; p.Ws = g.Wout; p.Cd = g.Cin; p.oH = g.Hin; p.oW = g.Win;
    p.S = 1; p.osy = p.osx = s; p.KK = KK; p.wm = KK; p.wk = g.Cin * KK; p.ncls = 0; p.rows_max = 1;
    int tap = 0;
    for (int ph = 0; ph < s; ph++)
        for (int pw = 0; pw < s; pw++) {
            if (ph >= g.Hin || pw >= g.Win) continue;
            CmClass &c = p.cls[p.ncls++];
            c.Hc = (g.Hin - ph + s - 1) / s; c.Wc = (g.Win - pw + s - 1) / s; c.oy0 = ph; c.ox0 = pw; c.tap0 = tap;
            const int rh = (ph + g.padU) % s, qh = (ph + g.padU) / s, rw = (pw + g.padL) % s, qw = (pw + g.padL) / s;
            int r0 = 127, r1 = -127, c0 = 127, c1 = -127;
            for (int kh = rh; kh < g.Hk; kh += s)
                for (int kw = rw; kw < g.Wk; kw += s) {
                    const int dr = qh - (kh - rh) / s, dc = qw - (kw - rw) / s;
                    p.dr[tap] = (signed char)dr; p.dc[tap] = (signed char)dc; p.widx[tap] = (unsigned char)(kh * g.Wk + kw);
                    r0 = std::min(r0, dr); r1 = std::max(r1, dr); c0 = std::min(c0, dc); c1 = std::max(c1, dc);
                    tap++;
                }
            c.ntaps = tap - c.tap0;
            if (!c.ntaps) { r0 = r1 = c0 = c1 = 0; }
            c.dr_min = r0; c.dc_min = c0; c.cols = c.Wc + c1 - c0; c.dW = cm_div(c.Wc); c.dcols = cm_div(c.cols);
            p.rows_max = std::max(p.rows_max, r1 - r0 + 1);
        }
    return conv_mma_dispatch<T>(p);
}
#define INST(T) template bool conv_mma_fw<T>(const ConvGeom &, const T *, const T *, const T *, T *); template bool conv_mma_ig<T>(const ConvGeom &, const T *, const T *, T *);
INST(float)
INST(__half)
#undef INST

// ---------------------------------------------------------------- weight gradient
// dW[co][ci][t] = sum over streams and output pixels of dY[co][p] X[ci][p S + t]: the contraction runs over pixels, both
// operands are read K-major out of the same channels-last staging (ldmatrix.trans / 4-byte loads at pixel addresses taken from
// a table, so taps, strides and row ends cost nothing).  CTA = WM x 16 output channels by WN x 8 NI input channels, all taps of
// its tap group in registers; WK warps share the pixels of a tile.  Every CTA leaves one partial dW, summed in CTA order by the
// reduction that the other weight-gradient kernels use.
struct CmWg {
    const void *x, *dy; float *part; void *dw;       // partial results per CTA, or (cluster kernel) the result
    int n, Ci, H, W, Co, Ho, Wo, S, KK, Wk, padU, padL, tap0, ntaps;
    int bn, st_tile, tiles, tiles_s, tiles_r, rows_max, cols, ci_tiles, steps, shares;       // tiles_r: tiles of a row longer than a tile
    CmDiv dW, dcols;
    uint32_t xpitch, dpitch, d_off, t_off, buf2;    // bytes: pixel of X / of dY; offsets of the dY tile, of the address tables, of the second tiles (0: none)
};

// One tile of output pixels: its first stream, first pixel, first row and column, the end of its pixels, the rows of X it needs.
struct CmWgTile { int s0, p0, i0, col_t, last, rows; };
__device__ __forceinline__ CmWgTile cm_wg_tile(const CmWg &p, int tile)
{
    const int P = p.Ho * p.Wo;
    const bool multi = P < p.bn, wide = p.Wo > p.bn;
    CmWgTile t;
    t.s0 = multi ? tile * p.st_tile : tile / p.tiles_s;
    const int ts = tile - (multi ? tile : t.s0 * p.tiles_s), row_t = wide ? ts / p.tiles_r : 0;
    t.col_t = wide ? (ts - row_t * p.tiles_r) * p.bn : 0;                                               // a tile within one long row
    t.p0 = multi ? 0 : wide ? row_t * p.Wo + t.col_t : ts * p.bn;
    t.i0 = wide ? row_t : cm_quot(t.p0, p.dW);
    t.last = multi ? P - 1 : wide ? t.p0 + min(p.bn, p.Wo - t.col_t) - 1 : min(t.p0 + p.bn, P) - 1;
    t.rows = ((wide ? t.i0 : cm_quot(t.last, p.dW)) - t.i0) * p.S + p.rows_max;
    return t;
}
// pixel q of the tile -> its bytes from the first pixel of the staged X (pixels without a value: that of pixel 0)
__device__ __forceinline__ int cm_wg_pixel(const CmWg &p, const CmWgTile &t, int q)
{
    const int P = p.Ho * p.Wo;
    const bool multi = P < p.bn, wide = p.Wo > p.bn;
    if (q >= (multi ? p.st_tile * P : t.last + 1 - t.p0)) q = 0;
    int st = 0, pp = t.p0 + q;
    if (multi) { st = q / P; pp = q - st * P; }
    const int i = wide ? t.i0 : cm_quot(pp, p.dW), j = pp - i * p.Wo - t.col_t;
    return ((st * t.rows + (i - t.i0) * p.S) * p.cols + j * p.S) * (int)p.xpitch;
}
// X and dY of a tile into shared memory (ASYNC: by copies that the caller waits for)
template <class T, int NT, int CI, int CO, bool ASYNC>
__device__ __forceinline__ void cm_wg_stage(const CmWg &p, const CmWgTile &t, uint32_t xs, uint32_t ds, int ci0, int co0, int warp)
{
    const int P = p.Ho * p.Wo;
    const bool multi = P < p.bn;
    const long long xplane = (long long)p.H * p.W;
    const T *xp = reinterpret_cast<const T *>(p.x) + ((long long)t.s0 * p.Ci + ci0) * xplane, *dp = reinterpret_cast<const T *>(p.dy) + ((long long)t.s0 * p.Co + co0) * P;
    const int st_n = multi ? p.st_tile : 1, run = multi ? P : p.bn, row0 = t.i0 * p.S - p.padU, col0 = t.col_t * p.S - p.padL, d_end = multi ? P : t.last + 1;
    const CmDiv drun = cm_div_dev(run);
    if constexpr (ASYNC) {
        cm_stage_async<NT>(xs, xp, st_n, p.n - t.s0, t.rows, p.cols, p.dcols, row0, col0, p.H, p.W, CI, p.Ci - ci0, (uint32_t)xplane, (uint32_t)(p.Ci * xplane), p.xpitch, warp);
        cm_stage_async<NT>(ds, dp, st_n, p.n - t.s0, 1, run, drun, 0, t.p0, 1, d_end, CO, p.Co - co0, (uint32_t)P, (uint32_t)(p.Co * P), p.dpitch, NT / 32 - 1 - warp);
    } else {
        cm_stage<T, NT>(xs, xp, st_n, p.n - t.s0, t.rows, p.cols, p.dcols, row0, col0, p.H, p.W, CI, p.Ci - ci0, (uint32_t)xplane, (uint32_t)(p.Ci * xplane), p.xpitch, warp);
        cm_stage<T, NT>(ds, dp, st_n, p.n - t.s0, 1, run, drun, 0, t.p0, 1, d_end, CO, p.Co - co0, (uint32_t)P, (uint32_t)(p.Co * P), p.dpitch, NT / 32 - 1 - warp);
    }
}

template <class T, int TAPS, int MI, int NI, int WM, int WN, int WK>
__global__ void __launch_bounds__(32 * WM * WN * WK, 2) conv_mma_wg_kernel(const __grid_constant__ CmWg p)
{
    // a first read of a parameter misses the constant cache, one after the other where an index depends on another one: all lines at once
#pragma unroll
    for (int i = 0; i < (int)(sizeof(CmWg) / 4); i += 16) asm volatile("" ::"r"(reinterpret_cast<const uint32_t *>(&p)[i]));
    constexpr int NT = 32 * WM * WN * WK, BN = 128;
    constexpr bool HALF = sizeof(T) == 2;
    constexpr int KS = HALF ? 16 : 8, STEPS = BN / KS;
    constexpr int KCH = STEPS / WK >= 2 ? 2 : 1;                            // k-steps per chain
    constexpr int CO = 16 * MI * WM, CI = 8 * NI * WN;
    extern __shared__ __align__(16) unsigned char cm_smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wk = warp / (WM * WN), wmn = warp % (WM * WN), wm = wmn / WN, wn = wmn % WN;
    const int ci0 = ((int)blockIdx.x % p.ci_tiles) * CI, co0 = ((int)blockIdx.x / p.ci_tiles) * CO;
    const uint32_t xs = (uint32_t)__cvta_generic_to_shared(cm_smem), ds = xs + p.d_off;
    int *table = reinterpret_cast<int *>(cm_smem + p.t_off);
    const int cols = p.cols;

    float acc[TAPS][MI][NI][4];
#pragma unroll
    for (int t = 0; t < TAPS; t++)
#pragma unroll
        for (int i = 0; i < MI; i++)
#pragma unroll
            for (int j = 0; j < NI; j++)
#pragma unroll
                for (int q = 0; q < 4; q++) acc[t][i][j][q] = 0.f;
    int toff[TAPS];
#pragma unroll
    for (int t = 0; t < TAPS; t++) { const int tt = p.tap0 + min(t, p.ntaps - 1); toff[t] = ((tt / p.Wk) * cols + tt % p.Wk) * (int)p.xpitch; }
    // pixels of the tile that no stream covers stay zero in the dY tile
    for (uint32_t e = tid * 16; e < BN * p.dpitch; e += NT * 16) {
        asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(ds + e), "r"(0) : "memory");
        if (p.buf2) asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(ds + p.buf2 + e), "r"(0) : "memory");
    }

    const int t_begin = (int)((long long)p.tiles * blockIdx.y / gridDim.y), t_end = (int)((long long)p.tiles * (blockIdx.y + 1) / gridDim.y);
    auto stage = [&](int tile, uint32_t buf, bool async) {
        const CmWgTile t = cm_wg_tile(p, tile);
        if (tid < BN) table[(buf ? BN : 0) + tid] = cm_wg_pixel(p, t, tid);
        if constexpr (!HALF)
            if (async) { cm_wg_stage<T, NT, CI, CO, true>(p, t, xs + buf, ds + buf, ci0, co0, warp); return; }
        cm_wg_stage<T, NT, CI, CO, false>(p, t, xs + buf, ds + buf, ci0, co0, warp);
    };
    // two sets of tiles (fp32): the next tile arrives by asynchronous copies while this one is multiplied
    const bool two = !HALF && p.buf2 != 0;
    uint32_t cur = 0;
    pdl_wait();
    __syncthreads();                                                       // the zeros of the dY tiles are in place
    if (two && t_begin < t_end) stage(t_begin, 0, true);
    for (int tile = t_begin; tile < t_end; tile++) {
        uint32_t off = 0;
        if (two) {
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncthreads();
            off = cur; cur ^= p.buf2;
            if (tile + 1 < t_end) stage(tile + 1, cur, true);
        } else {
            __syncthreads();
            stage(tile, 0, false);
            __syncthreads();
        }
        const int *tab = table + (off ? BN : 0);
        for (int s = wk * KCH; s < p.steps; s += WK * KCH) {
            uint32_t a[KCH][MI][4], al[HALF ? 1 : KCH][HALF ? 1 : MI][4], xa[KCH][HALF ? 1 : 2];
#pragma unroll
            for (int c = 0; c < KCH; c++) {
                const int k0 = (s + c) * KS;
                if constexpr (HALF) {
                    xa[c][0] = xs + off + (uint32_t)tab[k0 + (lane & 7) + ((lane >> 3) & 1) * 8] + (uint32_t)(wn * NI * 8 + (lane >> 4) * 8) * 2u;
#pragma unroll
                    for (int i = 0; i < MI; i++)
                        cm_ldsm_t(a[c][i], ds + off + (uint32_t)(k0 + (lane & 7) + (lane >> 4) * 8) * p.dpitch + (uint32_t)((wm * MI + i) * 16 + ((lane >> 3) & 1) * 8) * 2u);
                } else {
#pragma unroll
                    for (int h = 0; h < 2; h++) xa[c][h] = xs + off + (uint32_t)tab[k0 + (lane & 3) + 4 * h] + (uint32_t)(wn * NI * 8 + (lane >> 2)) * 4u;
#pragma unroll
                    for (int i = 0; i < MI; i++)
#pragma unroll
                        for (int q = 0; q < 4; q++)
                            tc::split_tf32_fast(__uint_as_float(cm_lds32(ds + off + (uint32_t)(k0 + (lane & 3) + (q >> 1) * 4) * p.dpitch + (uint32_t)((wm * MI + i) * 16 + (lane >> 2) + (q & 1) * 8) * 4u)), a[c][i][q], al[c][i][q]);
                }
            }
#pragma unroll
            for (int t = 0; t < TAPS; t++) {
                float tmp[MI][NI][4];
#pragma unroll
                for (int i = 0; i < MI; i++)
#pragma unroll
                    for (int j = 0; j < NI; j++)
#pragma unroll
                        for (int q = 0; q < 4; q++) tmp[i][j][q] = 0.f;
#pragma unroll
                for (int c = 0; c < KCH; c++) {
                    if constexpr (HALF) {
#pragma unroll
                        for (int j = 0; j < NI / 2; j++) {
                            uint32_t b[4];
                            cm_ldsm_t(b, xa[c][0] + toff[t] + j * 32u);
#pragma unroll
                            for (int i = 0; i < MI; i++) { cm_hmma(tmp[i][2 * j], a[c][i], b[0], b[1]); cm_hmma(tmp[i][2 * j + 1], a[c][i], b[2], b[3]); }
                        }
                    } else {
                        uint32_t bh[NI][2], bl[NI][2];
#pragma unroll
                        for (int j = 0; j < NI; j++)
#pragma unroll
                            for (int h = 0; h < 2; h++) tc::split_tf32_fast(__uint_as_float(cm_lds32(xa[c][h] + toff[t] + j * 32u)), bh[j][h], bl[j][h]);
#pragma unroll
                        for (int term = 0; term < 3; term++)
#pragma unroll
                            for (int j = 0; j < NI; j++)
#pragma unroll
                                for (int i = 0; i < MI; i++) cm_tmma(tmp[i][j], term == 0 ? al[c][i] : a[c][i], term == 1 ? bl[j][0] : bh[j][0], term == 1 ? bl[j][1] : bh[j][1]);
                    }
                }
#pragma unroll
                for (int i = 0; i < MI; i++)
#pragma unroll
                    for (int j = 0; j < NI; j++)
#pragma unroll
                        for (int q = 0; q < 4; q++) acc[t][i][j][q] += tmp[i][j][q];
            }
        }
    }
    // pixel shares of the warps meet in shared memory in the order of dW (taps innermost) and are added in warp order on the way
    // out: one barrier and contiguous stores (tap by tap it was two barriers each and every store its own sector)
    constexpr int RP = CI * TAPS + 4;
    float *red = reinterpret_cast<float *>(cm_smem);
    float *out = p.part + (size_t)blockIdx.y * p.Co * p.Ci * p.KK;
    __syncthreads();
#pragma unroll
    for (int t = 0; t < TAPS; t++)
#pragma unroll
        for (int i = 0; i < MI; i++)
#pragma unroll
            for (int j = 0; j < NI; j++)
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const int r = (wm * MI + i) * 16 + (lane >> 2) + (q >> 1) * 8, c = wn * NI * 8 + j * 8 + 2 * (lane & 3) + (q & 1);
                    red[(wk * CO + r) * RP + c * TAPS + t] = acc[t][i][j][q];
                }
    __syncthreads();
    for (int r = warp; r < CO; r += NT / 32) {
        if (co0 + r >= p.Co) break;
        float *row = out + ((long long)(co0 + r) * p.Ci + ci0) * p.KK + p.tap0;
        for (int e = lane; e < CI * TAPS; e += 32) {
            float v = red[r * RP + e];
#pragma unroll
            for (int k = 1; k < WK; k++) v += red[(k * CO + r) * RP + e];
            const int c = e / TAPS, t = e - c * TAPS;
            if (ci0 + c < p.Ci && t < p.ntaps) row[c * p.KK + t] = v;
        }
    }
}

// Few pixels (single streams).  What bounds these layers is the way from one launch to the next: the kernel above left one partial dW
// per CTA for a reduction of its own, gave half of its warps no pixels and wrote 72 accumulators a thread through shared memory.  Here
// the CTAs of one 16 x 16 channel tile are one cluster that shares the pixels, each of nine warps has filter taps of its own (fewer
// taps than warps: the warps share the pixels), and the cluster adds its results through distributed shared memory in rank order, so
// that no partial results and no second launch exist.
// Measured with the reduction, before and after: one stream of 16 -> 32 channels on 32 x 32 pixels 8.4 -> 5.9 us (fp16 7.3 -> 4.8), 2 -> 61
// on 33 x 46 with stride 2 8.6 -> 5.1, 48 -> 48 on 28 x 28 with 5 x 5 windows 27.1 -> 12.5 (three launches before).
static constexpr int CMC_NW = 9, CMC_TILE = 16, CMC_MAX = 16;
template <class T, int TPW>
__global__ void __launch_bounds__(32 * CMC_NW, 2) conv_mma_wg_cluster_kernel(const __grid_constant__ CmWg p)
{
#pragma unroll
    for (int i = 0; i < (int)(sizeof(CmWg) / 4); i += 16) asm volatile("" ::"r"(reinterpret_cast<const uint32_t *>(&p)[i]));
    constexpr int NT = 32 * CMC_NW, BN = 128, KS = sizeof(T) == 2 ? 16 : 8, KCH = 2;                    // KCH k-steps per chain
    constexpr bool HALF = sizeof(T) == 2;
    extern __shared__ __align__(16) unsigned char cm_smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rank = blockIdx.x, ranks = gridDim.x;                        // (the cluster is a row of the grid)
    const int co_t = (int)blockIdx.y / p.ci_tiles, ci0 = ((int)blockIdx.y - co_t * p.ci_tiles) * CMC_TILE, co0 = co_t * CMC_TILE;
    const uint32_t xs = (uint32_t)__cvta_generic_to_shared(cm_smem), ds = xs + p.d_off;
    int *table = reinterpret_cast<int *>(cm_smem + p.t_off);
    const int KK = p.KK, shares = p.shares, share = shares > 1 ? warp / KK : 0, tap = warp - share * KK;
    const int t_begin = p.tiles * rank / ranks, t_end = p.tiles * (rank + 1) / ranks;
    float acc[TPW][2][4] = {};
    int toff[TPW];
#pragma unroll
    for (int u = 0; u < TPW; u++) { const int t = min(tap + u * CMC_NW, KK - 1); toff[u] = ((t / p.Wk) * p.cols + t % p.Wk) * (int)p.xpitch; }
    // pixels of the tile that no stream covers are zero in the dY tile
    const int covered = p.Ho * p.Wo < p.bn ? p.st_tile * p.Ho * p.Wo : p.bn;
    for (uint32_t e = covered * p.dpitch + tid * 16; e < BN * p.dpitch; e += NT * 16) asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(ds + e), "r"(0) : "memory");
    pdl_wait();
    for (int tile = t_begin; tile < t_end; tile++) {
        if (tile > t_begin) __syncthreads();
        const CmWgTile t = cm_wg_tile(p, tile);
        cm_wg_stage<T, NT, CMC_TILE, CMC_TILE, false>(p, t, xs, ds, ci0, co0, warp);
        if (tid < BN) table[tid] = cm_wg_pixel(p, t, tid);
        __syncthreads();
        if (share >= shares) continue;
        for (int s = share * KCH; s < p.steps; s += shares * KCH) {
            uint32_t a[KCH][4], al[HALF ? 1 : KCH][4], xa[KCH][HALF ? 1 : 2];
#pragma unroll
            for (int c = 0; c < KCH; c++) {
                const int k0 = (s + c) * KS;
                if constexpr (HALF) {
                    xa[c][0] = xs + (uint32_t)table[k0 + (lane & 15)] + (uint32_t)(lane >> 4) * 16u;
                    cm_ldsm_t(a[c], ds + (uint32_t)(k0 + (lane & 7) + (lane >> 4) * 8) * p.dpitch + (uint32_t)((lane >> 3) & 1) * 16u);
                } else {
#pragma unroll
                    for (int h = 0; h < 2; h++) xa[c][h] = xs + (uint32_t)table[k0 + (lane & 3) + 4 * h] + (uint32_t)(lane >> 2) * 4u;
#pragma unroll
                    for (int q = 0; q < 4; q++)
                        tc::split_tf32_fast(__uint_as_float(cm_lds32(ds + (uint32_t)(k0 + (lane & 3) + (q >> 1) * 4) * p.dpitch + (uint32_t)((lane >> 2) + (q & 1) * 8) * 4u)), a[c][q], al[c][q]);
                }
            }
#pragma unroll
            for (int u = 0; u < TPW; u++) {
                if (u > 0 && tap + u * CMC_NW >= KK) break;
                float tmp[2][4] = {};
#pragma unroll
                for (int c = 0; c < KCH; c++) {
                    if constexpr (HALF) {
                        uint32_t b[4];
                        cm_ldsm_t(b, xa[c][0] + toff[u]);
                        cm_hmma(tmp[0], a[c], b[0], b[1]);
                        cm_hmma(tmp[1], a[c], b[2], b[3]);
                    } else {
                        uint32_t bh[2][2], bl[2][2];
#pragma unroll
                        for (int j = 0; j < 2; j++)
#pragma unroll
                            for (int h = 0; h < 2; h++) tc::split_tf32_fast(__uint_as_float(cm_lds32(xa[c][h] + toff[u] + j * 32u)), bh[j][h], bl[j][h]);
#pragma unroll
                        for (int term = 0; term < 3; term++)
#pragma unroll
                            for (int j = 0; j < 2; j++) cm_tmma(tmp[j], term == 0 ? al[c] : a[c], term == 1 ? bl[j][0] : bh[j][0], term == 1 ? bl[j][1] : bh[j][1]);
                    }
                }
#pragma unroll
                for (int j = 0; j < 2; j++)
#pragma unroll
                    for (int q = 0; q < 4; q++) acc[u][j][q] += tmp[j][q];
            }
        }
    }
    // the CTA's dW, rows of one output channel in memory order (taps innermost)
    const int cols = CMC_TILE * KK, RP = cols + 4;
    float *red = reinterpret_cast<float *>(cm_smem);
    __syncthreads();
    if (share < shares)
#pragma unroll
        for (int u = 0; u < TPW; u++) {
            if (tap + u * CMC_NW >= KK) break;
#pragma unroll
            for (int j = 0; j < 2; j++)
#pragma unroll
                for (int q = 0; q < 4; q++)
                    red[(share * CMC_TILE + (lane >> 2) + (q >> 1) * 8) * RP + (j * 8 + 2 * (lane & 3) + (q & 1)) * KK + tap + u * CMC_NW] = acc[u][j][q];
        }
    if (shares > 1) {
        __syncthreads();
        for (int e = tid; e < CMC_TILE * RP; e += NT) {
            float v = red[e];
            for (int k = 1; k < shares; k++) v += red[k * CMC_TILE * RP + e];
            red[e] = v;
        }
    }
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
    // a CTA adds 16 / ranks rows: 16 loads an element whatever the cluster's size, all on their way at once
    const int live = min(CMC_TILE, p.Ci - ci0) * KK, co_left = p.Co - co0;
    T *dw = reinterpret_cast<T *>(p.dw) + ((long long)co0 * p.Ci + ci0) * KK;
    auto remote = [&](int row, int e, int k) {
        uint32_t at; float v;
        asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(xs + (uint32_t)(row * RP + e) * 4u), "r"(k));
        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(at) : "memory");
        return v;
    };
    for (int e = tid; e < live; e += NT) {
        float v[CMC_MAX], sum = 0.f;
        if (ranks == CMC_MAX) {
            if (rank >= co_left) break;
#pragma unroll
            for (int k = 0; k < CMC_MAX; k++) v[k] = remote(rank, e, k);
#pragma unroll
            for (int k = 0; k < CMC_MAX; k++) sum += v[k];
            st(dw + (long long)rank * p.Ci * KK + e, sum);
        } else {
            const int rmask = ranks - 1;                                    // (a power of two)
#pragma unroll
            for (int q = 0; q < CMC_MAX; q++) v[q] = remote(rank + (q & ~rmask), e, q & rmask);
#pragma unroll
            for (int q = 0; q < CMC_MAX; q++) {
                sum += v[q];
                if ((q & rmask) == rmask) {
                    const int r = rank + (q & ~rmask);
                    if (r < co_left) st(dw + (long long)r * p.Ci * KK + e, sum);
                    sum = 0.f;
                }
            }
        }
    }
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");      // no CTA leaves while its sums are read
}

// Pixels per tile and their layout in shared memory (X, then dY), for `slots` CTAs that share the pixels.  false = not covered.
template <class T> static bool cm_wg_plan(CmWg &p, int CI, int CO, int slots, size_t &xb, size_t &db)
{
    constexpr int SZ = (int)sizeof(T), PAD = SZ == 2 ? 16 : 32;
    const int P = p.Ho * p.Wo, cols0 = p.cols;
    p.ci_tiles = ceil_div(p.Ci, CI);
    const long long stream_elements = (long long)p.Ci * p.H * p.W + (long long)p.Co * P;
    if (stream_elements >= (1ll << 25)) return false;                      // cm_streams
    auto tiles_of = [&](int bn) -> long long { return P < bn ? ceil_div(p.n, cm_streams(bn, P, p.n, stream_elements)) : p.Wo > bn ? (long long)p.n * p.Ho * ceil_div(p.Wo, bn) : (long long)p.n * ceil_div(P, bn); };
    // pixels per tile: what makes the fewest pixels of the longest CTA (planes and rounds come out even), halo rows included
    double best = 1e30;
    for (int bn = 128; bn >= 32; bn -= SZ == 2 ? 16 : 8) {
        const int halo = bn + 2 * std::min(p.Wo, bn) * (p.rows_max - 1) / 3;
        const double cost = (double)ceil_div(tiles_of(bn), slots) * halo;
        if (cost < 0.98 * best) { best = cost; p.bn = bn; }
    }
    const int bn = p.bn;
    p.st_tile = P < bn ? cm_streams(bn, P, p.n, stream_elements) : 1;
    const bool wide = p.Wo > bn;
    p.tiles_r = ceil_div(p.Wo, bn); p.tiles_s = wide ? p.Ho * p.tiles_r : ceil_div(P, bn);
    if (wide) { p.cols = (bn - 1) * p.S + cols0 - (p.Wo - 1) * p.S; p.dcols = cm_div(p.cols); }
    else if ((long long)P * p.Wo >= (1ll << 32)) return false;
    const long long tiles = tiles_of(bn);
    if (tiles >= (1 << 30)) return false;
    p.tiles = (int)tiles;
    p.steps = ceil_div(P < bn ? p.st_tile * P : bn, SZ == 2 ? 16 : 8);
    const int rows = (wide ? 0 : P < bn ? p.Ho - 1 : (bn + p.Wo - 2) / p.Wo) * p.S + p.rows_max;
    p.xpitch = CI * SZ + PAD; p.dpitch = CO * SZ + PAD;
    xb = ((size_t)p.st_tile * rows * p.cols * p.xpitch + 15) & ~(size_t)15; db = (size_t)128 * p.dpitch;
    p.d_off = (uint32_t)xb;
    return true;
}

// false: a cluster of more than eight CTAs, which not every device (or part of one) can place
template <class T, int TPW> static bool conv_mma_wg_cluster_launch(const CmWg &p, int ranks, size_t smem)
{
    static bool set = false, sixteen = false;
    if (!set) {
        cudaFuncSetAttribute(conv_mma_wg_cluster_kernel<T, TPW>, cudaFuncAttributeMaxDynamicSharedMemorySize, CM_SMEM_MAX);
        if (cudaFuncSetAttribute(conv_mma_wg_cluster_kernel<T, TPW>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess)
            sixteen = clusters_fit(conv_mma_wg_cluster_kernel<T, TPW>, 32 * CMC_NW, CM_SMEM_MAX, CMC_MAX);
        cudaGetLastError();
        set = true;
    }
    if (ranks > 8 && !sixteen) return false;
    TL_LAUNCH_CLUSTER((conv_mma_wg_cluster_kernel<T, TPW>), dim3(ranks, p.ci_tiles * ceil_div(p.Co, CMC_TILE)), 32 * CMC_NW, smem, ranks, p);
    return true;
}

template <class T, int TAPS, int MI, int NI, int WM, int WN, int WK> static bool conv_mma_wg_launch(CmWg &p, int part_groups, int *groups_out, bool dry)
{
    constexpr int BN = 128, SZ = (int)sizeof(T), CO = 16 * MI * WM, CI = 8 * NI * WN;
    const int ctiles = ceil_div(p.Ci, CI) * ceil_div(p.Co, CO);
    size_t xb, db;
    if (!cm_wg_plan<T>(p, CI, CO, std::max(1, std::min(2 * sm_count() / ctiles, part_groups)), xb, db)) return false;
    const bool two = SZ == 4 && 2 * (xb + db) + 8 * BN <= 110 * 1024;
    p.buf2 = two ? (uint32_t)(xb + db) : 0u; p.t_off = (uint32_t)((xb + db) * (two ? 2 : 1));
    const size_t smem = std::max((size_t)p.t_off + 8 * BN, (size_t)WK * CO * (CI * TAPS + 4) * 4);
    if (smem > CM_SMEM_MAX) return false;
    int groups = std::max(1, sm_count() * (smem <= 110 * 1024 ? 2 : 1) / ctiles);
    groups = std::min(std::min(groups, p.tiles), part_groups);
    *groups_out = groups;
    if (dry) return true;
    auto kern = conv_mma_wg_kernel<T, TAPS, MI, NI, WM, WN, WK>;
    static size_t attr = 0;
    if (smem > attr) { cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, CM_SMEM_MAX); attr = CM_SMEM_MAX; }
    for (p.tap0 = 0; p.tap0 < p.KK; p.tap0 += TAPS) {
        p.ntaps = std::min(TAPS, p.KK - p.tap0);
        TL_LAUNCH((conv_mma_wg_kernel<T, TAPS, MI, NI, WM, WN, WK>), dim3(ctiles, groups), 32 * WM * WN * WK, smem, p);
    }
    return true;
}

template <class T> static bool cm_wg_params(const ConvGeom &geom, const T *x, const T *dy, CmWg &p)
{
    const ConvGeom g = cm_flat(geom);
    const int KK = g.Hk * g.Wk;
    if (g.depthwise || gemm_path() == 1 || KK > CM_MAXTAPS || g.sh != g.sw || (long long)g.Hin * g.Win >= (1ll << 31)) return false;
    p = CmWg();
    p.x = x; p.dy = dy; p.n = g.n; p.Ci = g.Cin; p.H = g.Hin; p.W = g.Win; p.Co = g.Cout; p.Ho = g.Hout; p.Wo = g.Wout; p.S = g.sh;
    p.KK = KK; p.Wk = g.Wk; p.padU = g.padU; p.padL = g.padL; p.rows_max = g.Hk; p.cols = (g.Wout - 1) * g.sw + g.Wk; p.dW = cm_div(g.Wout); p.dcols = cm_div(p.cols);
    return true;
}

// Where it pays: while every CTA has an SM (a cluster of 16 needs most of a GPC, and 16 x 16 tiles read more per product than the kernel
// above: one stream of 64 -> 64 on 32 x 32, 256 CTAs, fp32 12.1 us against 9.4 there) and up to 2048 pixels (32 -> 32 on 64 x 64:
// 11.7 against 10.7; 32 -> 64 on two planes of 32 x 32, 9.6 against 9.8, is about where they meet) that every CTA stages at once (33 -> 27,
// 1 x 1, on 14 planes of 7 x 20, two tiles a CTA, fp16: 8.1 against 7.1).  Very few pixels under many channels
// leave the kernel above one partial result to write and read again per CTA: there up to eight CTAs an SM (256 -> 256 on 8 x 8
// 15.5 -> 11.4 us, 512 -> 512 on 4 x 4 37.1 -> 20.7), except for 1 x 1 windows (512 -> 512 on 4 x 4: 8.9 against 19.3).
template <class T> static bool cm_wg_cluster_plan(const ConvGeom &g, const T *x, const T *dy, CmWg &p, int &ranks, size_t &smem)
{
    size_t xb, db;
    if ((long long)g.n * g.Hout * g.Wout > CMC_MAX * 128 || !cm_wg_params(g, x, dy, p) || !cm_wg_plan<T>(p, CMC_TILE, CMC_TILE, CMC_MAX, xb, db)) return false;
    p.t_off = (uint32_t)(xb + db);
    p.shares = std::max(1, CMC_NW / p.KK);
    smem = std::max((size_t)p.t_off + 4 * 128, (size_t)p.shares * CMC_TILE * (CMC_TILE * p.KK + 4) * 4);
    for (ranks = 1; ranks < std::min(p.tiles, CMC_MAX);) ranks *= 2;
    const long long pixels = (long long)p.n * p.Ho * p.Wo, ctas = (long long)p.ci_tiles * ceil_div(p.Co, CMC_TILE) * ranks;
    return p.tiles <= CMC_MAX && smem <= CM_SMEM_MAX && (ctas <= sm_count() || (p.KK > 1 && pixels <= 64 && ctas <= 8ll * sm_count()));
}
template <class T> bool conv_mma_wg_cluster(const ConvGeom &g, const T *x, const T *dy, T *dw)
{
    CmWg p;
    int ranks;
    size_t smem;
    if (!cm_wg_cluster_plan<T>(g, x, dy, p, ranks, smem)) return false;
    p.dw = dw;
    const int tpw = ceil_div(p.KK, CMC_NW);
    return tpw <= 1 ? conv_mma_wg_cluster_launch<T, 1>(p, ranks, smem) : tpw <= 3 ? conv_mma_wg_cluster_launch<T, 3>(p, ranks, smem) : conv_mma_wg_cluster_launch<T, 6>(p, ranks, smem);
}
// fp16: in front of the tcgen05 kernel over slots, whose launch and reduction cost about 10 us at any size, while the products of a CTA
// are few (48 -> 48 on 28 x 28, 5 x 5: 8.6 us against 13.3; with 7 x 7 windows 16.6 against 15.5)
bool conv_mma_wg_cluster_first(const ConvGeom &g)
{
    CmWg p;
    int ranks;
    size_t smem;
    return cm_wg_cluster_plan<__half>(g, nullptr, nullptr, p, ranks, smem) && (long long)ranks * p.ci_tiles * ceil_div(p.Co, CMC_TILE) * p.KK * p.steps <= 100ll * sm_count();
}

// Partial results per CTA into `part`; false = geometry not covered.  dry_run: only the number of groups.
template <class T> bool conv_mma_wg(const ConvGeom &geom, const T *x, const T *dy, float *part, int part_groups, int *groups_out, bool dry)
{
    CmWg p;
    if (!cm_wg_params(geom, x, dy, p)) return false;
    const ConvGeom g = cm_flat(geom);
    const int KK = p.KK;
    p.part = part;
    if (KK == 1) {
        if (g.Cin > 32 && g.Cout > 16) return conv_mma_wg_launch<T, 1, 2, 4, 2, 2, 2>(p, part_groups, groups_out, dry);
        return conv_mma_wg_launch<T, 1, 1, 4, 2, 1, 4>(p, part_groups, groups_out, dry);
    }
    // channel tiles of 16 or 32 by what the layer has; the warps that a narrow layer leaves over share the pixels
    if (sizeof(T) == 2 && g.Cin > 16 && g.Cout > 32) return conv_mma_wg_launch<T, 9, 1, 2, 4, 2, 1>(p, part_groups, groups_out, dry);
    if (g.Cin > 16 && g.Cout > 16) return conv_mma_wg_launch<T, 9, 1, 2, 2, 2, 2>(p, part_groups, groups_out, dry);
    if (g.Cout > 16) return conv_mma_wg_launch<T, 9, 1, 2, 2, 1, 4>(p, part_groups, groups_out, dry);
    if (g.Cin > 16) return conv_mma_wg_launch<T, 9, 1, 2, 1, 2, 4>(p, part_groups, groups_out, dry);
    return conv_mma_wg_launch<T, 9, 1, 2, 1, 1, 8>(p, part_groups, groups_out, dry);
}
#define INST(T) template bool conv_mma_wg<T>(const ConvGeom &, const T *, const T *, float *, int, int *, bool); template bool conv_mma_wg_cluster<T>(const ConvGeom &, const T *, const T *, T *);
INST(float)
INST(__half)
#undef INST

} // namespace tl

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

// n / d for n, d < 2^16
struct CmDiv { uint32_t m; int d; };
static CmDiv cm_div(int d) { CmDiv r; r.d = d; r.m = d == 1 ? 0u : (uint32_t)(((1ull << 32) + d - 1) / d); return r; }
__device__ __forceinline__ CmDiv cm_div_dev(int d) { CmDiv r; r.d = d; r.m = d == 1 ? 0u : 0xFFFFFFFFu / (uint32_t)d + 1u; return r; }
__device__ __forceinline__ int cm_quot(int n, CmDiv d) { return d.m ? (int)__umulhi((uint32_t)n, d.m) : n; }

__device__ __forceinline__ void cm_ldsm(uint32_t (&r)[4], uint32_t addr) { asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr)); }
__device__ __forceinline__ void cm_ldsm_t(uint32_t (&r)[4], uint32_t addr) { asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr)); }
__device__ __forceinline__ void cm_hmma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void cm_tmma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t cm_lds32(uint32_t addr) { uint32_t v; asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr)); return v; }

// A patch of the source plane(s), channels-last: `streams` x rows x cols pixels of `chans` channels (a multiple of 8 fp16 / 4
// fp32; channels at or past c_left read as zero).  One item = one pixel x 16 bytes of channels: neighbouring threads take
// neighbouring pixels, so the per-channel loads are coalesced and the 16-byte store is conflict-free.
template <class T, int NT>
__device__ __forceinline__ void cm_stage(uint32_t sm, const T *src, int streams, int streams_left, int rows, int cols, CmDiv dcols, CmDiv drc, CmDiv dpix,
                                         int row0, int col0, int H, int W, int chans, int c_left, long long cstride, long long sstride, uint32_t pitch)
{
    constexpr int G = 16 / (int)sizeof(T);
    const int pix = streams * rows * cols, items = pix * (chans / G);
    for (int e = threadIdx.x; e < items; e += NT) {
        const int g = cm_quot(e, dpix), p = e - g * pix;                   // channel group, pixel of the patch
        const int st = cm_quot(p, drc), rc = p - st * drc.d, r = cm_quot(rc, dcols), c = rc - r * cols;
        const int h = row0 + r, w = col0 + c;
        const bool ok = st < streams_left && (unsigned)h < (unsigned)H && (unsigned)w < (unsigned)W;
        const T *s = src + st * sstride + (long long)(g * G) * cstride + (ok ? h * W + w : 0);
        uint32_t v[4];
        if constexpr (sizeof(T) == 2) {
            unsigned short u[8];
#pragma unroll
            for (int q = 0; q < 8; q++) u[q] = (ok && g * G + q < c_left) ? *reinterpret_cast<const unsigned short *>(s + q * cstride) : (unsigned short)0;
#pragma unroll
            for (int q = 0; q < 4; q++) v[q] = (uint32_t)u[2 * q] | ((uint32_t)u[2 * q + 1] << 16);
        } else {
#pragma unroll
            for (int q = 0; q < 4; q++) v[q] = (ok && g * G + q < c_left) ? *reinterpret_cast<const uint32_t *>(s + q * cstride) : 0u;
        }
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(sm + (uint32_t)p * pitch + (uint32_t)g * 16u), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
    }
}

// ---------------------------------------------------------------- forward and input gradient
// dst[m][oy0 + i osy][ox0 + j osx] = sum over taps t and source channels k of src[k][i S + dr_t][j S + dc_t] W[m][k][t].
// Forward: S = the stride, one class.  Input gradient: a class per parity (oy0, ox0) of the input pixels (osy = osx = the
// stride, S = 1), whose taps are the ones that reach that parity; the weights are read with the channel roles swapped.
struct CmClass { int Hc, Wc, oy0, ox0, tap0, ntaps, dr_min, dc_min, cols; CmDiv dW, dcols; };
struct CmFwd {
    const void *src, *w, *bias; void *dst;
    int n, Cs, Hs, Ws, Cd, oH, oW, S, osy, osx, KK;
    int wm, wk;                              // weight index = m * wm + k * wk + tap
    int ncls; CmClass cls[9];
    signed char dr[CM_MAXTAPS], dc[CM_MAXTAPS]; unsigned char widx[CM_MAXTAPS];
    int st_tile;                             // streams per tile (planes smaller than a tile), else 1
    int CKS, groups, cblk, resident;         // channels staged at a time, how often, k-steps per chain; weights loaded once per CTA
    uint32_t pitch, wpitch, w_off;           // bytes: pixel, weight row; offset of the weights behind the patch
    int rows_max;
};

template <class T, int MT, int WM, int WN, int WK, int BN>
__global__ void __launch_bounds__(32 * WM * WN * WK, 2) conv_mma_kernel(const __grid_constant__ CmFwd p)
{
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
    const int tiles_s = P < BN ? 1 : (P + BN - 1) / BN;                     // tiles of one stream
    const int tiles = (P < BN ? (p.n + p.st_tile - 1) / p.st_tile : p.n * tiles_s);
    if ((int)blockIdx.x >= tiles) return;

    for (int t = tid; t < p.KK; t += NT) tap_of[t] = -1;
    __syncthreads();
    for (int t = tid; t < ntaps; t += NT) {
        tap_off[t] = ((p.dr[c.tap0 + t] - c.dr_min) * c.cols + (p.dc[c.tap0 + t] - c.dc_min)) * (int)p.pitch;
        tap_of[p.widx[c.tap0 + t]] = t;
    }
    __syncthreads();

    // weights of channels k0 .. k0 + kc as [tap][BM][wpitch], one contiguous source run per row (or per contraction channel)
    auto load_weights = [&](int k0, int kc) {
        const T *w = reinterpret_cast<const T *>(p.w);
        const CmDiv dKK = cm_div_dev(p.KK);
        if (p.wk == p.KK) {
            const int run = kc * p.KK, live = min(kc, p.Cs - k0) * p.KK;
            for (int m = warp; m < BM; m += NT / 32) {
                const T *row = w + (long long)(m0 + m) * p.wm + (long long)k0 * p.KK;
                const bool in = m0 + m < p.Cd;
                for (int e = lane; e < run; e += 32) {
                    const int k = cm_quot(e, dKK), t = tap_of[e - k * p.KK];
                    const T v = (in && e < live) ? row[e] : T(0.f);
                    if (t >= 0) *reinterpret_cast<T *>(cm_smem + p.w_off + (size_t)((t * BM + m) * (int)p.wpitch + k * SZ)) = v;
                }
            }
        } else {
            const int run = BM * p.KK, live = min(BM, p.Cd - m0) * p.KK;
            for (int k = warp; k < kc; k += NT / 32) {
                const T *row = w + (long long)(k0 + k) * p.wk + (long long)m0 * p.KK;
                const bool in = k0 + k < p.Cs;
                for (int e = lane; e < run; e += 32) {
                    const int m = cm_quot(e, dKK), t = tap_of[e - m * p.KK];
                    const T v = (in && e < live) ? row[e] : T(0.f);
                    if (t >= 0) *reinterpret_cast<T *>(cm_smem + p.w_off + (size_t)((t * BM + m) * (int)p.wpitch + k * SZ)) = v;
                }
            }
        }
    };
    if (p.resident) load_weights(0, p.groups * p.CKS);

    const CmDiv dcols = c.dcols, dW = c.dW;
    const long long src_plane = (long long)p.Hs * p.Ws, dst_plane = (long long)p.oH * p.oW;

    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int s0 = P < BN ? tile * p.st_tile : tile / tiles_s, p0 = P < BN ? 0 : (tile % tiles_s) * BN;
        const int st_n = P < BN ? p.st_tile : 1;
        const int i0 = cm_quot(p0, dW);
        const int live = P < BN ? min(st_n, p.n - s0) * P : min(BN, P - p0);        // output pixels of this tile
        const int last = P < BN ? P - 1 : min(p0 + BN, P) - 1;
        const int rows = (cm_quot(last, dW) - i0) * p.S + p.rows_max;               // rows_max: rows that one output row needs
        // start addresses (in the patch) of the pixels this lane supplies fragments for
        constexpr int NB = HALF ? N8 / 2 : N8;
        uint32_t pix[NB];
#pragma unroll
        for (int j = 0; j < NB; j++) {
            int q = wn * TN + (HALF ? j * 16 + (lane & 7) + ((lane >> 4) & 1) * 8 : j * 8 + (lane >> 2));
            if (q >= live) q = 0;
            int st = 0, pp = p0 + q;
            if (P < BN) { st = q / P; pp = q - st * P; }
            const int i = cm_quot(pp, dW), jj = pp - i * c.Wc;
            pix[j] = patch + (uint32_t)(((st * rows + (i - i0) * p.S) * c.cols + jj * p.S) * (int)p.pitch) + (HALF ? (uint32_t)((lane >> 3) & 1) * 16u : (uint32_t)(lane & 3) * 4u);
        }
        float acc[MT][N8][4];
#pragma unroll
        for (int i = 0; i < MT; i++)
#pragma unroll
            for (int j = 0; j < N8; j++)
#pragma unroll
                for (int q = 0; q < 4; q++) acc[i][j][q] = 0.f;

        for (int g = 0; g < p.groups; g++) {
            __syncthreads();                                                        // the patch (and the weights) are free again
            const int k0 = g * p.CKS;
            if (!p.resident) load_weights(k0, p.CKS);
            const CmDiv drc = cm_div_dev(rows * c.cols), dpix = cm_div_dev(st_n * rows * c.cols);
            cm_stage<T, NT>(patch, reinterpret_cast<const T *>(p.src) + ((long long)s0 * p.Cs + k0) * src_plane, st_n, p.n - s0, rows, c.cols, dcols, drc, dpix,
                            i0 * p.S + c.dr_min, c.dc_min, p.Hs, p.Ws, p.CKS, p.Cs - k0, src_plane, (long long)p.Cs * src_plane, p.pitch);
            __syncthreads();
            const uint32_t wg = wsm + (uint32_t)(p.resident ? k0 * SZ : 0);
            const int nck = p.CKS / CK, nblk = (nck + p.cblk - 1) / p.cblk;
            for (int u = wk; u < ntaps * nblk; u += WK) {
                const int t = nblk == 1 ? u : u / nblk, ck0 = nblk == 1 ? 0 : (u - t * nblk) * p.cblk, ck1 = min(nck, ck0 + p.cblk);
                const uint32_t toff = (uint32_t)tap_off[t];
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
#pragma unroll
                        for (int j = 0; j < N8; j++) {
                            uint32_t bh0, bl0, bh1, bl1;
                            tc::split_tf32_fast(__uint_as_float(cm_lds32(pix[j] + toff + ck * 32u)), bh0, bl0);
                            tc::split_tf32_fast(__uint_as_float(cm_lds32(pix[j] + toff + ck * 32u + 16u)), bh1, bl1);
#pragma unroll
                            for (int i = 0; i < MT; i++) { cm_tmma(tmp[i][j], al[i], bh0, bh1); cm_tmma(tmp[i][j], ah[i], bl0, bl1); cm_tmma(tmp[i][j], ah[i], bh0, bh1); }
                        }
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
            if (wk > 0) continue;
        }
        // results: a lane holds pixel pairs of two rows (output channels) per 16 x 8 fragment
        T *dst = reinterpret_cast<T *>(p.dst);
        const T *bias = reinterpret_cast<const T *>(p.bias);
#pragma unroll
        for (int j = 0; j < N8; j++) {
            const int q0 = wn * TN + 8 * j + 2 * (lane & 3);
            long long off[2];
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int q = min(q0 + h, live - 1);
                int st = 0, pp = p0 + q;
                if (P < BN) { st = q / P; pp = q - st * P; }
                const int i = cm_quot(pp, dW), jj = pp - i * c.Wc;
                off[h] = ((long long)(s0 + st) * p.Cd) * dst_plane + (long long)(c.oy0 + i * p.osy) * p.oW + c.ox0 + jj * p.osx;
            }
#pragma unroll
            for (int i = 0; i < MT; i++)
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int m = m0 + wm * 16 * MT + i * 16 + (lane >> 2) + h * 8;
                    if (m >= p.Cd || q0 >= live) continue;
                    const float bv = bias ? ld(bias + m) : 0.f;
                    const float v0 = acc[i][j][2 * h] + bv, v1 = acc[i][j][2 * h + 1] + bv;
                    T *d0 = dst + off[0] + m * dst_plane;
                    if (q0 + 1 < live && off[1] == off[0] + 1 && (((uintptr_t)d0) & (2 * SZ - 1)) == 0) {
                        if constexpr (HALF) *reinterpret_cast<__half2 *>(d0) = __floats2half2_rn(v0, v1);
                        else *reinterpret_cast<float2 *>(d0) = make_float2(v0, v1);
                    } else {
                        st(d0, v0);
                        if (q0 + 1 < live) st(dst + off[1] + m * dst_plane, v1);
                    }
                }
        }
    }
}

template <class T, int MT, int WM, int WN, int WK, int BN> static bool conv_mma_launch(CmFwd &p, int cpad, bool dry)
{
    constexpr int CK = sizeof(T) == 2 ? 16 : 8, SZ = (int)sizeof(T), BM = 16 * MT * WM;
    // the largest patch over the classes: streams x rows x cols
    long long pix = 0; int taps = 0, tiles_max = 0; p.st_tile = 1;
    const int P0 = p.cls[0].Hc * p.cls[0].Wc;                              // class 0 has the most pixels
    if (P0 < BN) p.st_tile = std::max(1, std::min(BN / P0, p.n));
    for (int i = 0; i < p.ncls; i++) {
        const CmClass &c = p.cls[i];
        const int P = c.Hc * c.Wc;
        const int rows = (P < BN ? c.Hc - 1 : (BN + c.Wc - 2) / c.Wc) * p.S + p.rows_max;
        pix = std::max(pix, (long long)p.st_tile * rows * c.cols);
        taps = std::max(taps, c.ntaps);
        tiles_max = std::max(tiles_max, P < BN ? ceil_div(p.n, p.st_tile) : (int)std::min<long long>((long long)p.n * ceil_div(P, BN), 1 << 30));
    }
    const size_t red = WK > 1 ? (size_t)(WK - 1) * WM * WN * MT * (BN / WN / 8) * 512 : 0;
    auto plan = [&](int cks, bool resident, size_t limit) {
        p.CKS = cks; p.groups = ceil_div(cpad, cks); p.resident = resident;
        p.pitch = (uint32_t)(cks * SZ + 16); p.wpitch = (uint32_t)((resident ? p.groups * cks : cks) * SZ + 16);
        const size_t pb = std::max<size_t>(((size_t)pix * p.pitch + 15) & ~(size_t)15, red);
        p.w_off = (uint32_t)pb;
        return pb + (size_t)taps * BM * p.wpitch <= limit;
    };
    // everything resident in half of an SM's shared memory if it fits (two CTAs overlap staging and arithmetic), else fewer
    // channels at a time, else all of it, else weights reloaded with every group of channels
    bool ok = false;
    for (size_t limit : {(size_t)110 * 1024, (size_t)CM_SMEM_MAX}) {
        for (int parts = 1; !ok && parts <= cpad / CK; parts *= 2) ok = plan(ceil_div(ceil_div(cpad, parts), CK) * CK, true, limit);
        if (ok) break;
        for (int parts = 1; !ok && parts <= cpad / CK; parts *= 2) ok = plan(ceil_div(ceil_div(cpad, parts), CK) * CK, false, limit);
        if (ok) break;
    }
    if (!ok) return false;
    if (dry) return true;
    const int nck = p.CKS / CK;
    p.cblk = std::min(nck, 16);
    while (WK > 1 && p.cblk > 1 && taps * ceil_div(nck, p.cblk) < 2 * WK) p.cblk = (p.cblk + 1) / 2;
    const size_t smem = p.w_off + (size_t)taps * BM * p.wpitch;
    auto kern = conv_mma_kernel<T, MT, WM, WN, WK, BN>;
    static size_t attr = 0;
    if (smem > attr) { cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, CM_SMEM_MAX); attr = CM_SMEM_MAX; }
    const int co_tiles = ceil_div(p.Cd, BM);
    const int slots = std::max(1, sm_count() * (smem <= 110 * 1024 ? 2 : 1) / (co_tiles * p.ncls));
    const int rounds = ceil_div(tiles_max, slots), gx = ceil_div(tiles_max, rounds);
    TL_LAUNCH((conv_mma_kernel<T, MT, WM, WN, WK, BN>), dim3(gx, co_tiles, p.ncls), 32 * WM * WN * WK, smem, p);
    return true;
}

template <class T> static bool conv_mma_dispatch(CmFwd &p)
{
    constexpr int CK = sizeof(T) == 2 ? 16 : 8;
    const int cpad = ceil_div(p.Cs, CK) * CK;
    long long tiles = 0;                                                   // 128-pixel tiles
    for (int i = 0; i < p.ncls; i++) tiles += ((long long)p.n * p.cls[i].Hc * p.cls[i].Wc + 127) / 128;
    // Few tiles (single streams): 16 x 32 result tiles whose taps and channels are dealt to four warps each, so that a layer of
    // 32 channels on 32 x 32 pixels still occupies 64 CTAs; otherwise 128 pixels by 16, 32 or 64 channels.
    if (tiles * ceil_div(p.Cd, p.Cd > 32 ? 64 : 32) < sm_count()) return conv_mma_launch<T, 1, 1, 2, 4, 32>(p, cpad, false);
    if (p.Cd > 32) return conv_mma_launch<T, 2, 2, 4, 1, 128>(p, cpad, false) || conv_mma_launch<T, 1, 1, 8, 1, 128>(p, cpad, false);
    if (p.Cd > 16) return conv_mma_launch<T, 2, 1, 8, 1, 128>(p, cpad, false) || conv_mma_launch<T, 1, 1, 8, 1, 128>(p, cpad, false);
    return conv_mma_launch<T, 1, 1, 8, 1, 128>(p, cpad, false);
}

// false = not covered, nothing launched
template <class T> bool conv_mma_fw(const ConvGeom &g, const T *x, const T *w, const T *bias, T *y)
{
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
template <class T> bool conv_mma_ig(const ConvGeom &g, const T *dy, const T *w, T *dx)
{
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
    const void *x, *dy; float *part;
    int n, Ci, H, W, Co, Ho, Wo, S, KK, Wk, padU, padL, tap0, ntaps;
    int st_tile, tiles, tiles_s, rows_max, cols, ci_tiles, steps;
    CmDiv dW, dcols;
    uint32_t xpitch, dpitch, d_off, t_off;      // bytes: pixel of X / of dY; offsets of the dY tile and of the address table
};

template <class T, int TAPS, int MI, int NI, int WM, int WN, int WK>
__global__ void __launch_bounds__(32 * WM * WN * WK, 2) conv_mma_wg_kernel(const __grid_constant__ CmWg p)
{
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
    const int P = p.Ho * p.Wo, cols = p.cols;
    const bool multi = P < BN;
    const CmDiv dW = p.dW, dcols = p.dcols;

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
    for (uint32_t e = tid * 16; e < BN * p.dpitch; e += NT * 16) asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(ds + e), "r"(0) : "memory");

    const int per = (p.tiles + gridDim.y - 1) / gridDim.y, t_begin = blockIdx.y * per, t_end = min(p.tiles, t_begin + per);
    const long long xplane = (long long)p.H * p.W;
    for (int tile = t_begin; tile < t_end; tile++) {
        const int s0 = multi ? tile * p.st_tile : tile / p.tiles_s, p0 = multi ? 0 : (tile % p.tiles_s) * BN;
        const int st_n = multi ? p.st_tile : 1;
        const int i0 = cm_quot(p0, dW), last = multi ? P - 1 : min(p0 + BN, P) - 1;
        const int rows = (cm_quot(last, dW) - i0) * p.S + p.rows_max;
        __syncthreads();
        if (tid < BN) {
            const int live = multi ? st_n * P : last + 1 - p0, q = tid < live ? tid : 0;
            int st = 0, pp = p0 + q;
            if (multi) { st = q / P; pp = q - st * P; }
            const int i = cm_quot(pp, dW), j = pp - i * p.Wo;
            table[tid] = ((st * rows + (i - i0) * p.S) * cols + j * p.S) * (int)p.xpitch;
        }
        const CmDiv drc = cm_div_dev(rows * cols), dpix = cm_div_dev(st_n * rows * cols);
        cm_stage<T, NT>(xs, reinterpret_cast<const T *>(p.x) + ((long long)s0 * p.Ci + ci0) * xplane, st_n, p.n - s0, rows, cols, dcols, drc, dpix,
                        i0 * p.S - p.padU, -p.padL, p.H, p.W, CI, p.Ci - ci0, xplane, (long long)p.Ci * xplane, p.xpitch);
        const int run = multi ? P : BN;
        const CmDiv drun = cm_div_dev(run), dall = cm_div_dev(st_n * run);
        cm_stage<T, NT>(ds, reinterpret_cast<const T *>(p.dy) + ((long long)s0 * p.Co + co0) * P, st_n, p.n - s0, 1, run, drun, drun, dall,
                        0, p0, 1, P, CO, p.Co - co0, P, (long long)p.Co * P, p.dpitch);
        __syncthreads();
        for (int s = wk * KCH; s < p.steps; s += WK * KCH) {
            uint32_t a[KCH][MI][4], al[HALF ? 1 : KCH][HALF ? 1 : MI][4], xa[KCH][HALF ? 1 : 2];
#pragma unroll
            for (int c = 0; c < KCH; c++) {
                const int k0 = (s + c) * KS;
                if constexpr (HALF) {
                    xa[c][0] = xs + (uint32_t)table[k0 + (lane & 7) + ((lane >> 3) & 1) * 8] + (uint32_t)(wn * NI * 8 + (lane >> 4) * 8) * 2u;
#pragma unroll
                    for (int i = 0; i < MI; i++)
                        cm_ldsm_t(a[c][i], ds + (uint32_t)(k0 + (lane & 7) + (lane >> 4) * 8) * p.dpitch + (uint32_t)((wm * MI + i) * 16 + ((lane >> 3) & 1) * 8) * 2u);
                } else {
#pragma unroll
                    for (int h = 0; h < 2; h++) xa[c][h] = xs + (uint32_t)table[k0 + (lane & 3) + 4 * h] + (uint32_t)(wn * NI * 8 + (lane >> 2)) * 4u;
#pragma unroll
                    for (int i = 0; i < MI; i++)
#pragma unroll
                        for (int q = 0; q < 4; q++)
                            tc::split_tf32_fast(__uint_as_float(cm_lds32(ds + (uint32_t)(k0 + (lane & 3) + (q >> 1) * 4) * p.dpitch + (uint32_t)((wm * MI + i) * 16 + (lane >> 2) + (q & 1) * 8) * 4u)), a[c][i][q], al[c][i][q]);
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
#pragma unroll
                        for (int j = 0; j < NI; j++) {
                            uint32_t bh0, bl0, bh1, bl1;
                            tc::split_tf32_fast(__uint_as_float(cm_lds32(xa[c][0] + toff[t] + j * 32u)), bh0, bl0);
                            tc::split_tf32_fast(__uint_as_float(cm_lds32(xa[c][1] + toff[t] + j * 32u)), bh1, bl1);
#pragma unroll
                            for (int i = 0; i < MI; i++) { cm_tmma(tmp[i][j], al[c][i], bh0, bh1); cm_tmma(tmp[i][j], a[c][i], bl0, bl1); cm_tmma(tmp[i][j], a[c][i], bh0, bh1); }
                        }
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
    // pixel shares of the warps added in warp order, one tap at a time; then this CTA's partial
    float *red = reinterpret_cast<float *>(cm_smem);
    float *out = p.part + (size_t)blockIdx.y * p.Co * p.Ci * p.KK;
#pragma unroll
    for (int t = 0; t < TAPS; t++) {
        __syncthreads();
#pragma unroll
        for (int i = 0; i < MI; i++)
#pragma unroll
            for (int j = 0; j < NI; j++)
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const int r = (wm * MI + i) * 16 + (lane >> 2) + (q >> 1) * 8, c = wn * NI * 8 + j * 8 + 2 * (lane & 3) + (q & 1);
                    red[(wk * CO + r) * CI + c] = acc[t][i][j][q];
                }
        __syncthreads();
        if (t < p.ntaps)
            for (int e = tid; e < CO * CI; e += NT) {
                const int r = e / CI, c = e % CI;
                float v = red[e];
#pragma unroll
                for (int k = 1; k < WK; k++) v += red[k * CO * CI + e];
                if (co0 + r < p.Co && ci0 + c < p.Ci) out[((long long)(co0 + r) * p.Ci + ci0 + c) * p.KK + p.tap0 + t] = v;
            }
    }
}

template <class T, int TAPS, int MI, int NI, int WM, int WN, int WK> static bool conv_mma_wg_launch(CmWg &p, int part_groups, int *groups_out, bool dry)
{
    constexpr int BN = 128, SZ = (int)sizeof(T), CO = 16 * MI * WM, CI = 8 * NI * WN, PAD = SZ == 2 ? 16 : 32;
    const int P = p.Ho * p.Wo;
    p.st_tile = P < BN ? std::max(1, std::min(BN / P, p.n)) : 1;
    p.tiles_s = ceil_div(P, BN);
    const long long tiles = P < BN ? ceil_div(p.n, p.st_tile) : (long long)p.n * p.tiles_s;
    if (tiles >= (1 << 30)) return false;
    p.tiles = (int)tiles;
    p.steps = ceil_div(P < BN ? p.st_tile * P : BN, SZ == 2 ? 16 : 8);
    const int rows = (P < BN ? p.Ho - 1 : (BN + p.Wo - 2) / p.Wo) * p.S + p.rows_max;
    p.xpitch = CI * SZ + PAD; p.dpitch = CO * SZ + PAD;
    const size_t xb = ((size_t)p.st_tile * rows * p.cols * p.xpitch + 15) & ~(size_t)15, db = (size_t)BN * p.dpitch;
    p.d_off = (uint32_t)xb; p.t_off = (uint32_t)(xb + db);
    const size_t smem = std::max(xb + db + BN * 4, (size_t)WK * CO * CI * 4);
    if (smem > CM_SMEM_MAX) return false;
    p.ci_tiles = ceil_div(p.Ci, CI);
    const int ctiles = p.ci_tiles * ceil_div(p.Co, CO);
    int groups = std::max(1, sm_count() * (smem <= 110 * 1024 ? 2 : 1) / ctiles);
    groups = std::min(std::min(groups, p.tiles), part_groups);
    groups = ceil_div(p.tiles, ceil_div(p.tiles, groups));
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

// Partial results per CTA into `part`; false = geometry not covered.  dry_run: only the number of groups.
template <class T> bool conv_mma_wg(const ConvGeom &g, const T *x, const T *dy, float *part, int part_groups, int *groups_out, bool dry)
{
    const int KK = g.Hk * g.Wk;
    if (g.depthwise || gemm_path() == 1 || KK > CM_MAXTAPS || g.sh != g.sw || (long long)g.Hin * g.Win >= (1ll << 31)) return false;
    CmWg p;
    p.x = x; p.dy = dy; p.part = part; p.n = g.n; p.Ci = g.Cin; p.H = g.Hin; p.W = g.Win; p.Co = g.Cout; p.Ho = g.Hout; p.Wo = g.Wout; p.S = g.sh;
    p.KK = KK; p.Wk = g.Wk; p.padU = g.padU; p.padL = g.padL; p.rows_max = g.Hk; p.cols = (g.Wout - 1) * g.sw + g.Wk; p.dW = cm_div(g.Wout); p.dcols = cm_div(p.cols);
    if (KK == 1) {
        if (g.Cin > 32 && g.Cout > 16) return conv_mma_wg_launch<T, 1, 2, 4, 2, 2, 2>(p, part_groups, groups_out, dry);
        return conv_mma_wg_launch<T, 1, 1, 4, 2, 1, 4>(p, part_groups, groups_out, dry);
    }
    // channel tiles of 16 or 32 by what the layer has; the warps that a narrow layer leaves over share the pixels
    if (g.Cin > 16 && g.Cout > 16) return conv_mma_wg_launch<T, 9, 1, 2, 2, 2, 2>(p, part_groups, groups_out, dry);
    if (g.Cout > 16) return conv_mma_wg_launch<T, 9, 1, 2, 2, 1, 4>(p, part_groups, groups_out, dry);
    if (g.Cin > 16) return conv_mma_wg_launch<T, 9, 1, 2, 1, 2, 4>(p, part_groups, groups_out, dry);
    return conv_mma_wg_launch<T, 9, 1, 2, 1, 1, 8>(p, part_groups, groups_out, dry);
}
#define INST(T) template bool conv_mma_wg<T>(const ConvGeom &, const T *, const T *, float *, int, int *, bool);
INST(float)
INST(__half)
#undef INST

} // namespace tl

// Depthwise convolution, one filter per channel [ref: lib/sources/pulp_conv_naive_fp32.c:29,113,153].  The layer does nine multiply-adds per
// value read, so nothing may be read twice from HBM.  3 x 3 filters with stride 1 work in registers (the strips below).  For the others, on planes
// that fit shared memory, a CTA stages whole planes of one or more
// (stream, channel) pairs with their zero border once (coalesced, each value read once from HBM), and every window is then
// read from shared memory without bounds checks.  64 channels of 28 x 28 x 64 streams, fp32 (25.7 MB per pass): forward 45 us
// and input gradient 92 us with one bounds-checked global read per tap; 145 us for the weight gradient, which ran one CTA per
// (channel, tap).
#include "tl_kernels.h"
#include "tl_reduce.cuh"
#include <algorithm>

namespace tl {

// A launch gets 48 KB of shared memory without asking, and the kernel's static arrays count: up to 800 bytes here (the sums of 25
// taps over eight warps).  Above this the limit is raised for the kernel first.
static constexpr size_t DW_DEFAULT_SMEM = 48 * 1024 - 8 * 25 * sizeof(float);
template <class K> static void dw_allow(K kernel, size_t smem) { if (smem > DW_DEFAULT_SMEM) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); }

struct DwDiv { uint32_t m; int d; };
static DwDiv dw_div(int d) { DwDiv r; r.d = d; r.m = d == 1 ? 0u : 0xFFFFFFFFu / (uint32_t)d + 1u; return r; }
__device__ __forceinline__ int dw_quot(int n, DwDiv d) { return d.m ? (int)__umulhi((uint32_t)n, d.m) : n; }

struct DwParams {
    int C, planes, G;                            // channels, stream-channel pairs, pairs per CTA
    int Hs, Ws, Ho, Wo, sh, sw, Hk, Wk, r0, c0;  // source plane, result plane, origin of the staged window in the source
    int PH, PW, flip;
    DwDiv dPW, dP, dWo, dO;                      // staged width, staged plane, result width, result plane
};

// result[ho][wo] = sum over taps src[ho sh + kh + r0][wo sw + kw + c0] w[kh][kw]; flip: the filter rotated by 180 degrees (the
// input gradient of a stride-1 layer is the same sum over dY)
template <class T, int K>
__global__ void __launch_bounds__(256) dw_plane_kernel(const __grid_constant__ DwParams p, const T *__restrict__ src, const T *__restrict__ w, T *__restrict__ dst)
{
    pdl_wait();
    extern __shared__ float dw_smem[];
    const int KH = K ? K : p.Hk, KW = K ? K : p.Wk, KK = KH * KW;
    const int pl0 = blockIdx.x * p.G, np = min(p.G, p.planes - pl0), P = p.PH * p.PW, O = p.Ho * p.Wo;
    float *win = dw_smem, *ws = dw_smem + p.G * P;
    const T *s0 = src + (long long)pl0 * p.Hs * p.Ws;
#pragma unroll 4
    for (int e = threadIdx.x; e < np * P; e += 256) {
        const int g = dw_quot(e, p.dP), rc = e - g * P, r = dw_quot(rc, p.dPW), c = rc - r * p.PW;
        const int h = r + p.r0, x = c + p.c0;
        win[e] = ld0((unsigned)h < (unsigned)p.Hs && (unsigned)x < (unsigned)p.Ws, s0 + (g * p.Hs + h) * p.Ws + x);
    }
    for (int e = threadIdx.x; e < np * KK; e += 256) {
        const int g = e / KK, t = e - g * KK;
        ws[e] = ld(w + (long long)((pl0 + g) % p.C) * KK + (p.flip ? KK - 1 - t : t));
    }
    __syncthreads();
    T *d0 = dst + (long long)pl0 * O;
    for (int e = threadIdx.x; e < np * O; e += 256) {
        const int g = dw_quot(e, p.dO), ij = e - g * O, i = dw_quot(ij, p.dWo), j = ij - i * p.Wo;
        const float *b = win + g * P + i * p.sh * p.PW + j * p.sw, *wp = ws + g * KK;
        float acc = 0.f;
        if constexpr (K > 0) {
#pragma unroll
            for (int kh = 0; kh < K; kh++)
#pragma unroll
                for (int kw = 0; kw < K; kw++) acc = fmaf(wp[kh * K + kw], b[kh * p.PW + kw], acc);
        } else {
            for (int kh = 0; kh < KH; kh++)
                for (int kw = 0; kw < KW; kw++) acc = fmaf(wp[kh * KW + kw], b[kh * p.PW + kw], acc);
        }
        st(d0 + e, acc);
    }
}

// dW of one channel: the CTA walks its share of the streams; every thread keeps all taps of its pixels, the CTA's sums leave as
// one partial per (stream share, channel) and are added in order by the reduction of the other weight gradients.
template <class T, int K>
__global__ void __launch_bounds__(256) dw_wg_plane_kernel(const __grid_constant__ DwParams p, const T *__restrict__ x, const T *__restrict__ dy, float *__restrict__ part, int n)
{
    pdl_wait();
    extern __shared__ float dw_smem[];
    __shared__ float red[8][K * K];
    const int ch = blockIdx.x, P = p.PH * p.PW, O = p.Ho * p.Wo;
    const int per = (n + gridDim.y - 1) / gridDim.y, s_begin = blockIdx.y * per, s_end = min(n, s_begin + per);
    float acc[K * K];
#pragma unroll
    for (int t = 0; t < K * K; t++) acc[t] = 0.f;
    for (int s = s_begin; s < s_end; s += p.G) {
        const int ns = min(p.G, s_end - s);
        __syncthreads();
#pragma unroll 4
        for (int e = threadIdx.x; e < ns * P; e += 256) {
            const int g = dw_quot(e, p.dP), rc = e - g * P, r = dw_quot(rc, p.dPW), c = rc - r * p.PW;
            const int h = r + p.r0, xx = c + p.c0;
            dw_smem[e] = ld0((unsigned)h < (unsigned)p.Hs && (unsigned)xx < (unsigned)p.Ws, x + (((long long)(s + g) * p.C + ch) * p.Hs + h) * p.Ws + xx);
        }
        __syncthreads();
#pragma unroll 2
        for (int e = threadIdx.x; e < ns * O; e += 256) {
            const int g = dw_quot(e, p.dO), ij = e - g * O, i = dw_quot(ij, p.dWo), j = ij - i * p.Wo;
            const float d = ld(dy + ((long long)(s + g) * p.C + ch) * O + ij);
            const float *b = dw_smem + g * P + i * p.sh * p.PW + j * p.sw;
#pragma unroll
            for (int kh = 0; kh < K; kh++)
#pragma unroll
                for (int kw = 0; kw < K; kw++) acc[kh * K + kw] = fmaf(d, b[kh * p.PW + kw], acc[kh * K + kw]);
        }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int t = 0; t < K * K; t++) { const float v = warp_sum(acc[t]); if (lane == 0) red[warp][t] = v; }
    __syncthreads();
    if (threadIdx.x < K * K) {
        float v = red[0][threadIdx.x];
#pragma unroll
        for (int q = 1; q < 8; q++) v += red[q][threadIdx.x];
        part[((long long)blockIdx.y * p.C + ch) * K * K + threadIdx.x] = v;
    }
}

__device__ __forceinline__ void dw_st4(float *p, const float (&v)[4]) { *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]); }
__device__ __forceinline__ void dw_st4(__half *p, const float (&v)[4])
{
    const __half2 a = __floats2half2_rn(v[0], v[1]), b = __floats2half2_rn(v[2], v[3]);
    *reinterpret_cast<uint2 *>(p) = make_uint2(*reinterpret_cast<const uint32_t *>(&a), *reinterpret_cast<const uint32_t *>(&b));
}

// A thread has V neighbouring columns of a strip of up to R rows of one plane: every row of the source is read once per strip (its
// neighbours' columns come from L1), straight into registers, all rows of the strip in flight together, with no shared memory, no
// zero border and no barrier.  V = 4: rows of whole 16-byte groups (8 in fp16) and one column of padding.  Six CTAs of 128 threads fit an SM (two of 256 left a
// wave half empty at 4096 planes of 28 x 28: 6.6 / 6.2 us, fp16 6.1 / 5.0).  Staging planes in shared
// memory with a zero border was bound by that memory's pipe, half of its wavefronts bank conflicts; now it is the loads: 25.7 MB in
// 6.2 us of the layer above (4.1 TB/s), and with rows of odd lengths, three 4-byte loads a value, their issue.  us, staged / here, forward and both
// gradients: 64 channels of 28 x 28 x 64 streams 10.4 / 6.2 and 24.6 / 14.6 (fp16 10.0 / 5.0, 23.3 / 12.6); 64 of 112 x 112 x 4 16.0 / 5.5, 36.9 / 13.7;
// 48 of 27 x 33 x 100 15.1 / 13.1, 36.1 / 30.4; planes of one stream as before, by their launches (3.2 / 3.0).  Strips of eight rows instead of
// four change nothing in the weight gradient.
struct Dw3Strip {
    int C, planes, G, Hs, Ws, Ho, Wo, padU, padL, flip;
    int strips, rows, cols;                      // strips of a plane, rows of a strip, threads of a row
    DwDiv dPer, dCols;
};
__device__ __forceinline__ float4 dw_ld4_0(bool ok, const float *p) { float4 v = make_float4(0.f, 0.f, 0.f, 0.f); if (ok) v = *reinterpret_cast<const float4 *>(p); return v; }
__device__ __forceinline__ float4 dw_ld4_0(bool ok, const __half *p)
{
    uint2 u = make_uint2(0u, 0u);
    if (ok) u = *reinterpret_cast<const uint2 *>(p);
    const float2 a = __half22float2(*reinterpret_cast<const __half2 *>(&u.x)), b = __half22float2(*reinterpret_cast<const __half2 *>(&u.y));
    return make_float4(a.x, a.y, b.x, b.y);
}
// rows h0 .. h0 + R + 1 of a plane, `need` of them, the V + 2 columns around result column V j
template <class T, int V, int R> __device__ __forceinline__ void dw3_strip_load(const Dw3Strip &p, const T *s, int h0, int need, int j, float (&v)[R + 2][V + 2])
{
#pragma unroll
    for (int r = 0; r < R + 2; r++) {
        const bool ok = r < need && (unsigned)(h0 + r) < (unsigned)p.Hs;
        const T *row = s + (h0 + r) * p.Ws;
        if constexpr (V == 4) {
            const float4 m = dw_ld4_0(ok && 4 * j < p.Ws, row + 4 * j);
            v[r][0] = ld0(ok && j > 0 && 4 * j - 1 < p.Ws, row + 4 * j - 1); v[r][1] = m.x; v[r][2] = m.y; v[r][3] = m.z; v[r][4] = m.w;
            v[r][5] = ld0(ok && 4 * j + 4 < p.Ws, row + 4 * j + 4);
        } else {
#pragma unroll
            for (int k = 0; k < 3; k++) v[r][k] = ld0(ok && (unsigned)(j - p.padL + k) < (unsigned)p.Ws, row + j - p.padL + k);
        }
    }
}
template <class T, int V, int R>
__global__ void __launch_bounds__(128, 6) dw3_strip_kernel(const __grid_constant__ Dw3Strip p, const T *__restrict__ src, const T *__restrict__ w, T *__restrict__ dst)
{
    pdl_wait();
    const int pl0 = blockIdx.x * p.G, np = min(p.G, p.planes - pl0), per = p.strips * p.cols, c0 = pl0 % p.C;
    for (int e = blockIdx.y * 128 + threadIdx.x; e < np * per; e += 128 * gridDim.y) {
        const int g = p.G == 1 ? 0 : dw_quot(e, p.dPer), q = e - g * per, strip = dw_quot(q, p.dCols), j = q - strip * p.cols, i0 = strip * p.rows, rows = min(p.rows, p.Ho - i0);
        int c = c0 + g;
        while (c >= p.C) c -= p.C;
        float wv[9], v[R + 2][V + 2];
#pragma unroll
        for (int t = 0; t < 9; t++) wv[t] = ld(w + (long long)c * 9 + (p.flip ? 8 - t : t));
        dw3_strip_load<T, V, R>(p, src + (long long)(pl0 + g) * p.Hs * p.Ws, i0 - p.padU, rows + 2, j, v);
        T *o = dst + (long long)(pl0 + g) * p.Ho * p.Wo + (long long)i0 * p.Wo + V * j;
#pragma unroll
        for (int r = 0; r < R; r++, o += p.Wo) {
            if (r >= rows) break;
            float acc[V];
#pragma unroll
            for (int k = 0; k < V; k++) acc[k] = 0.f;
#pragma unroll
            for (int t = 0; t < 9; t++)
#pragma unroll
                for (int k = 0; k < V; k++) acc[k] = fmaf(wv[t], v[r + t / 3][k + t % 3], acc[k]);
            if constexpr (V == 4) dw_st4(o, acc);
            else st(o, acc[0]);
        }
    }
}
template <class T, int V, int R>
__global__ void __launch_bounds__(128, 4) dw3_strip_wg_kernel(const __grid_constant__ Dw3Strip p, const T *__restrict__ x, const T *__restrict__ dy, float *__restrict__ part, int n)
{
    pdl_wait();
    __shared__ float red[4][9];
    const int ch = blockIdx.x, per = p.strips * p.cols;
    const int s_begin = (int)((long long)n * blockIdx.y / gridDim.y), s_end = (int)((long long)n * (blockIdx.y + 1) / gridDim.y);
    float acc[9];
#pragma unroll
    for (int t = 0; t < 9; t++) acc[t] = 0.f;
    int s = s_begin, q = threadIdx.x;
    while (q >= per) { q -= per; s++; }
    while (s < s_end) {
        const int strip = dw_quot(q, p.dCols), j = q - strip * p.cols, i0 = strip * p.rows, rows = min(p.rows, p.Ho - i0);
        const long long pl = (long long)s * p.C + ch;
        const T *dp = dy + pl * p.Ho * p.Wo + (long long)i0 * p.Wo + V * j;
        float d[R][V], v[R + 2][V + 2];
#pragma unroll
        for (int r = 0; r < R; r++, dp += p.Wo) {
            if constexpr (V == 4) { const float4 t = dw_ld4_0(r < rows, dp); d[r][0] = t.x; d[r][1] = t.y; d[r][2] = t.z; d[r][3] = t.w; }
            else d[r][0] = ld0(r < rows, dp);
        }
        dw3_strip_load<T, V, R>(p, x + pl * p.Hs * p.Ws, i0 - p.padU, rows + 2, j, v);
        // a strip's own sum first: short chains, which the longer ones of a thread then add up
#pragma unroll
        for (int t = 0; t < 9; t++) {
            float sum = 0.f;
#pragma unroll
            for (int r = 0; r < R; r++)
#pragma unroll
                for (int k = 0; k < V; k++) sum = fmaf(d[r][k], r < rows ? v[r + t / 3][k + t % 3] : 0.f, sum);
            acc[t] += sum;
        }
        q += 128;
        while (q >= per) { q -= per; s++; }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int t = 0; t < 9; t++) { const float v = warp_sum(acc[t]); if (lane == 0) red[warp][t] = v; }
    __syncthreads();
    if (threadIdx.x < 9) part[((long long)blockIdx.y * p.C + ch) * 9 + threadIdx.x] = ((red[0][threadIdx.x] + red[1][threadIdx.x]) + red[2][threadIdx.x]) + red[3][threadIdx.x];
}
// V of the strips; 0: not covered
static int dw3_strip(const ConvGeom &g, Dw3Strip &p, const void *src, const void *dst, int esize, bool ig, int R)
{
    if (g.Hk != 3 || g.Wk != 3 || g.sh != 1 || g.sw != 1) return 0;
    p.C = g.Cin; p.planes = g.n * g.Cin; p.flip = ig;
    p.Hs = ig ? g.Hout : g.Hin; p.Ws = ig ? g.Wout : g.Win; p.Ho = ig ? g.Hin : g.Hout; p.Wo = ig ? g.Win : g.Wout;
    p.padU = ig ? 2 - g.padU : g.padU; p.padL = ig ? 2 - g.padL : g.padL;
    if ((long long)g.n * g.Cin >= (1ll << 31) || (long long)p.Hs * p.Ws >= (1ll << 24) || (long long)p.Ho * p.Wo >= (1ll << 24)) return 0;
    const int V = p.padL == 1 && p.Ws % 4 == 0 && p.Wo % 4 == 0 && ((uintptr_t)src | (uintptr_t)dst) % (4 * esize) == 0 ? 4 : 1;
    p.cols = p.Wo / V; p.strips = ceil_div(p.Ho, R); p.rows = ceil_div(p.Ho, p.strips); p.strips = ceil_div(p.Ho, p.rows);
    if ((long long)p.strips * p.cols * p.cols >= (1ll << 32)) return 0;     // (exact quotients)
    p.dPer = dw_div(p.strips * p.cols); p.dCols = dw_div(p.cols);
    return V;
}

static bool dw_window(const ConvGeom &g, DwParams &p, bool ig)
{
    p.C = g.Cin; p.planes = g.n * g.Cin; p.flip = ig; p.Hk = g.Hk; p.Wk = g.Wk;
    if (ig) {
        if (g.sh != 1 || g.sw != 1) return false;
        p.Hs = g.Hout; p.Ws = g.Wout; p.Ho = g.Hin; p.Wo = g.Win; p.sh = p.sw = 1; p.r0 = -(g.Hk - 1 - g.padU); p.c0 = -(g.Wk - 1 - g.padL);
    } else {
        p.Hs = g.Hin; p.Ws = g.Win; p.Ho = g.Hout; p.Wo = g.Wout; p.sh = g.sh; p.sw = g.sw; p.r0 = -g.padU; p.c0 = -g.padL;
    }
    p.PH = (p.Ho - 1) * p.sh + g.Hk; p.PW = (p.Wo - 1) * p.sw + g.Wk;
    if ((long long)g.n * g.Cin >= (1ll << 31) || (long long)p.PH * p.PW > 24 * 1024) return false;     // 96 KB of shared memory
    p.dPW = dw_div(p.PW); p.dP = dw_div(p.PH * p.PW); p.dWo = dw_div(p.Wo); p.dO = dw_div(p.Ho * p.Wo);
    return true;
}

// forward and stride-1 input gradient; false = not covered
template <class T> bool dw_planes(const ConvGeom &g, const T *src, const T *w, T *dst, bool ig)
{
    Dw3Strip t;
    if (const int V = dw3_strip(g, t, src, dst, (int)sizeof(T), ig, 8)) {
        const int per = t.strips * t.cols;
        // planes of a CTA: up to two rounds of its threads, as full as they get, fewer where that would leave SMs idle; the rounds are CTAs of
        // their own while SMs are
        const int most = std::max(1, std::min(per >= 4096 ? 1 : per >= 256 ? 2 : 256 / per, t.planes / (4 * sm_count())));
        double full = 0.0;
        t.G = 1;
        for (int G = 1; G <= most; G++) {
            const double f = (double)(G * per) / (ceil_div(G * per, 128) * 128);
            if (f > full + 0.01) { full = f; t.G = G; }
        }
        const int groups = ceil_div(t.planes, t.G);
        const dim3 grid(groups, std::max(1, std::min(ceil_div(t.G * per, 128), 6 * sm_count() / groups)));
        if (V == 4) TL_LAUNCH((dw3_strip_kernel<T, 4, 8>), grid, 128, 0, t, src, w, dst);
        else TL_LAUNCH((dw3_strip_kernel<T, 1, 8>), grid, 128, 0, t, src, w, dst);
        return true;
    }
    DwParams p;
    if (!dw_window(g, p, ig)) return false;
    const int P = p.PH * p.PW, O = p.Ho * p.Wo, KK = g.Hk * g.Wk;
    // about a thousand results per CTA (four per thread), fewer when that would leave SMs idle
    p.G = std::max(1, std::min(1024 / O, p.planes / (2 * sm_count())));
    while (p.G > 1 && (size_t)p.G * (P + KK) * 4 > 48 * 1024) p.G--;
    const size_t smem = (size_t)p.G * (P + KK) * 4;
    const int grid = ceil_div(p.planes, p.G);
#define TL_DW(KV)                                                             \
    do {                                                                      \
        dw_allow(dw_plane_kernel<T, KV>, smem);                               \
        TL_LAUNCH((dw_plane_kernel<T, KV>), grid, 256, smem, p, src, w, dst); \
    } while (0)
    if (g.Hk == 3 && g.Wk == 3) TL_DW(3); else if (g.Hk == 5 && g.Wk == 5) TL_DW(5); else TL_DW(0);
#undef TL_DW
    return true;
}
// partial weight gradients [groups][C][K*K]; 3 x 3 and 5 x 5 filters.  dry: only the number of groups
template <class T> bool dw_wg_planes(const ConvGeom &g, const T *x, const T *dy, float *part, int &groups, bool dry)
{
    Dw3Strip t;
    if (const int V = dw3_strip(g, t, x, dy, (int)sizeof(T), false, 4)) {
        // One wave of the four CTAs that fit an SM (two waves and a bit: 17.1 us for both gradients of 64 channels of 28 x 28 x 64, 14.6 so) while
        // that is two CTAs a channel.  From 297 channels on it would be one, half of the CTA slots empty or a second wave of few: about a
        // wave and a half there (us, one / two / three CTAs a channel: 300 channels of 28 x 28 x 64 37.2 / 34.4 / 29.8; 384 38.8 / 38.1 / 33.1; 512 of
        // 14 x 14 x 64 27.3 / 23.5 / 24.6; 600 32.7 / 28.8 / 28.1; 650 of 14 x 14 x 32 18.3 / 16.6 / 17.7; 960 of 7 x 7 x 64 15.0 / 14.7 / 16.1;
        // little work, 400 of 7 x 7 x 16, 5.7 / 5.8 / 5.8; below: 256 of 28 x 28 x 64 30.8 / 23.5 / 25.9)
        groups = std::max(1, std::min(g.Cin > 2 * sm_count() ? ceil_div(6 * sm_count(), g.Cin) : 4 * sm_count() / g.Cin, g.n));
        if (dry) return true;
        const dim3 grid(g.Cin, groups);
        if (V == 4) TL_LAUNCH((dw3_strip_wg_kernel<T, 4, 4>), grid, 128, 0, t, x, dy, part, g.n);
        else TL_LAUNCH((dw3_strip_wg_kernel<T, 1, 4>), grid, 128, 0, t, x, dy, part, g.n);
        return true;
    }
    DwParams p;
    if (g.Hk != g.Wk || (g.Hk != 3 && g.Hk != 5) || !dw_window(g, p, false)) return false;
    const int P = p.PH * p.PW, O = p.Ho * p.Wo;
    groups = std::max(1, std::min(ceil_div(4 * sm_count(), g.Cin), g.n));
    groups = ceil_div(g.n, ceil_div(g.n, groups));
    if (dry) return true;
    p.G = std::max(1, std::min(1024 / O, ceil_div(g.n, groups)));
    while (p.G > 1 && (size_t)p.G * P * 4 > 48 * 1024) p.G--;
    const size_t smem = (size_t)p.G * P * 4;
    const dim3 grid(g.Cin, groups);
#define TL_DW(KV)                                                                     \
    do {                                                                              \
        dw_allow(dw_wg_plane_kernel<T, KV>, smem);                                    \
        TL_LAUNCH((dw_wg_plane_kernel<T, KV>), grid, 256, smem, p, x, dy, part, g.n); \
    } while (0)
    if (g.Hk == 3) TL_DW(3); else TL_DW(5);
#undef TL_DW
    return true;
}
#define INST(T) template bool dw_planes<T>(const ConvGeom &, const T *, const T *, T *, bool); template bool dw_wg_planes<T>(const ConvGeom &, const T *, const T *, float *, int &, bool);
INST(float)
INST(__half)
#undef INST

} // namespace tl

// Depthwise convolution, one filter per channel [ref: lib/sources/pulp_conv_naive_fp32.c:29,113,153], for planes that fit
// shared memory.  The layer does nine multiply-adds per value read, so nothing may be read twice from HBM.  A CTA stages whole planes of one or more
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

// ---------------------------------------------------------------- 3 x 3, stride 1
// The common case with four neighbouring results per thread: a window row of six values serves four results (two or three
// shared loads per twelve multiply-adds instead of one per multiply-add), the filter sits in registers, and rows of whole
// 16-byte groups (8 bytes in fp16) move as vectors.  Shared-memory rows hold image column w at index 4 + w between zero columns.
// What bounds it is the shared-memory pipe: busy 88 % of the cycles of a forward pass of the layer above (11 us by itself), half of
// its wavefronts bank conflicts.
template <class T> struct DwVec;
template <> struct DwVec<float> { typedef float4 V; };
template <> struct DwVec<__half> { typedef uint2 V; };
__device__ __forceinline__ float4 dw_ld4(const float *p) { return *reinterpret_cast<const float4 *>(p); }
__device__ __forceinline__ float4 dw_ld4(const __half *p)
{
    const uint2 u = *reinterpret_cast<const uint2 *>(p);
    const float2 a = __half22float2(*reinterpret_cast<const __half2 *>(&u.x)), b = __half22float2(*reinterpret_cast<const __half2 *>(&u.y));
    return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ void dw_st4(float *p, const float (&v)[4]) { *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]); }
__device__ __forceinline__ void dw_st4(__half *p, const float (&v)[4])
{
    const __half2 a = __floats2half2_rn(v[0], v[1]), b = __floats2half2_rn(v[2], v[3]);
    *reinterpret_cast<uint2 *>(p) = make_uint2(*reinterpret_cast<const uint32_t *>(&a), *reinterpret_cast<const uint32_t *>(&b));
}

struct Dw3Params {
    int C, planes, G, Hs, Ws, Ho, Wo, padU, padL, flip;
    int PH, PW, W4, O4, vec_s, vec_o;            // staged rows, floats per staged row, quads per source row / result row, vector access
    DwDiv dW4, dWs, dRow, dO4;                   // dRow: quads (or values) of a source plane
};
// one plane group of the source into shared memory (the zero border is already there)
template <class T, int NT> __device__ __forceinline__ void dw3_stage(const Dw3Params &p, const T *src, int np, float *win, long long plane_step)
{
    const int P = p.PH * p.PW;
    if (p.vec_s) {
        const int per = p.Hs * p.W4;
#pragma unroll 2
        for (int e = threadIdx.x; e < np * per; e += NT) {
            const int g = dw_quot(e, p.dRow), q = e - g * per, r = dw_quot(q, p.dW4), c4 = q - r * p.W4;
            *reinterpret_cast<float4 *>(win + g * P + (r + p.padU) * p.PW + 4 + 4 * c4) = dw_ld4(src + g * plane_step + r * p.Ws + 4 * c4);
        }
    } else {
        const int per = p.Hs * p.Ws;
#pragma unroll 4
        for (int e = threadIdx.x; e < np * per; e += NT) {
            const int g = dw_quot(e, p.dRow), q = e - g * per, r = dw_quot(q, p.dWs), c = q - r * p.Ws;
            win[g * P + (r + p.padU) * p.PW + 4 + c] = ld(src + g * plane_step + q);
        }
    }
}
// the six window values that four neighbouring results need from one row
template <int PADL> __device__ __forceinline__ void dw3_row(const float *row, float (&v)[6])
{
    if constexpr (PADL == 1) {
        const float4 m = *reinterpret_cast<const float4 *>(row + 4);
        v[0] = row[3]; v[1] = m.x; v[2] = m.y; v[3] = m.z; v[4] = m.w; v[5] = row[8];
    } else {
#pragma unroll
        for (int k = 0; k < 6; k++) v[k] = row[4 - PADL + k];
    }
}
template <class T, int PADL>
__global__ void __launch_bounds__(128) dw3_kernel(const __grid_constant__ Dw3Params p, const T *__restrict__ src, const T *__restrict__ w, T *__restrict__ dst)
{
    pdl_wait();
    extern __shared__ __align__(16) float dw_smem[];
    const int P = p.PH * p.PW, pl0 = blockIdx.x * p.G, np = min(p.G, p.planes - pl0), O = p.Ho * p.Wo, per = p.Ho * p.O4;
    float *ws = dw_smem + p.G * P;
    for (int e = threadIdx.x; e < np * P / 4; e += 128) reinterpret_cast<float4 *>(dw_smem)[e] = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int e = threadIdx.x; e < np * 9; e += 128) { const int g = e / 9, t = e - 9 * g; ws[e] = ld(w + (long long)((pl0 + g) % p.C) * 9 + (p.flip ? 8 - t : t)); }
    __syncthreads();
    dw3_stage<T, 128>(p, src + (long long)pl0 * p.Hs * p.Ws, np, dw_smem, (long long)p.Hs * p.Ws);
    __syncthreads();
    T *d0 = dst + (long long)pl0 * O;
    for (int e = threadIdx.x; e < np * per; e += 128) {
        const int g = p.G == 1 ? 0 : dw_quot(e, p.dO4), q = e - g * per, i = q / p.O4, j4 = q - i * p.O4;
        const float *b = dw_smem + g * P + i * p.PW + 4 * j4, *wp = ws + g * 9;
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int kh = 0; kh < 3; kh++) {
            float v[6];
            dw3_row<PADL>(b + kh * p.PW, v);
#pragma unroll
            for (int kw = 0; kw < 3; kw++) {
                const float wv = wp[kh * 3 + kw];
#pragma unroll
                for (int k = 0; k < 4; k++) acc[k] = fmaf(wv, v[k + kw], acc[k]);
            }
        }
        T *o = d0 + (long long)g * O + i * p.Wo + 4 * j4;
        if (p.vec_o) dw_st4(o, acc);
        else {
#pragma unroll
            for (int k = 0; k < 4; k++) if (4 * j4 + k < p.Wo) st(o + k, acc[k]);
        }
    }
}
template <class T, int PADL>
__global__ void __launch_bounds__(128) dw3_wg_kernel(const __grid_constant__ Dw3Params p, const T *__restrict__ x, const T *__restrict__ dy, float *__restrict__ part, int n)
{
    pdl_wait();
    extern __shared__ __align__(16) float dw_smem[];
    __shared__ float red[4][9];
    const int ch = blockIdx.x, P = p.PH * p.PW, O = p.Ho * p.Wo, per = p.Ho * p.O4;
    const int s_begin = (int)((long long)n * blockIdx.y / gridDim.y), s_end = (int)((long long)n * (blockIdx.y + 1) / gridDim.y);
    for (int e = threadIdx.x; e < p.G * P / 4; e += 128) reinterpret_cast<float4 *>(dw_smem)[e] = make_float4(0.f, 0.f, 0.f, 0.f);
    float acc[9];
#pragma unroll
    for (int t = 0; t < 9; t++) acc[t] = 0.f;
    for (int s = s_begin; s < s_end; s += p.G) {
        const int ns = min(p.G, s_end - s);
        __syncthreads();
        dw3_stage<T, 128>(p, x + ((long long)s * p.C + ch) * p.Hs * p.Ws, ns, dw_smem, (long long)p.C * p.Hs * p.Ws);
        __syncthreads();
#pragma unroll 2
        for (int e = threadIdx.x; e < ns * per; e += 128) {
            const int g = p.G == 1 ? 0 : dw_quot(e, p.dO4), q = e - g * per, i = q / p.O4, j4 = q - i * p.O4;
            const T *dp = dy + ((long long)(s + g) * p.C + ch) * O + i * p.Wo + 4 * j4;
            float d[4];
            if (p.vec_o) { const float4 t = dw_ld4(dp); d[0] = t.x; d[1] = t.y; d[2] = t.z; d[3] = t.w; }
            else {
#pragma unroll
                for (int k = 0; k < 4; k++) d[k] = ld0(4 * j4 + k < p.Wo, dp + k);
            }
            const float *b = dw_smem + g * P + i * p.PW + 4 * j4;
#pragma unroll
            for (int kh = 0; kh < 3; kh++) {
                float v[6];
                dw3_row<PADL>(b + kh * p.PW, v);
#pragma unroll
                for (int kw = 0; kw < 3; kw++)
#pragma unroll
                    for (int k = 0; k < 4; k++) acc[kh * 3 + kw] = fmaf(d[k], v[k + kw], acc[kh * 3 + kw]);
            }
        }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int t = 0; t < 9; t++) { const float v = warp_sum(acc[t]); if (lane == 0) red[warp][t] = v; }
    __syncthreads();
    if (threadIdx.x < 9) part[((long long)blockIdx.y * p.C + ch) * 9 + threadIdx.x] = ((red[0][threadIdx.x] + red[1][threadIdx.x]) + red[2][threadIdx.x]) + red[3][threadIdx.x];
}

static bool dw3_params(const ConvGeom &g, Dw3Params &p, const void *src, const void *dst, int esize, bool ig)
{
    if (g.Hk != 3 || g.Wk != 3 || g.sh != 1 || g.sw != 1) return false;
    p.C = g.Cin; p.planes = g.n * g.Cin; p.flip = ig;
    p.Hs = ig ? g.Hout : g.Hin; p.Ws = ig ? g.Wout : g.Win; p.Ho = ig ? g.Hin : g.Hout; p.Wo = ig ? g.Win : g.Wout;
    p.padU = ig ? 2 - g.padU : g.padU; p.padL = ig ? 2 - g.padL : g.padL;
    if (p.padU < 0 || p.padL < 0 || p.padL > 2 || p.padU > 2 || (long long)g.n * g.Cin >= (1ll << 31)) return false;
    p.PH = std::max(p.Ho + 2, p.Hs + p.padU); p.O4 = ceil_div(p.Wo, 4); p.W4 = p.Ws / 4;
    p.PW = std::max(4 * p.O4 + 12, 4 + (p.Ws + 3) / 4 * 4);
    if ((long long)p.PH * p.PW > 12 * 1024) return false;                  // 48 KB of planes
    p.vec_s = p.Ws % 4 == 0 && ((uintptr_t)src) % (4 * esize) == 0; p.vec_o = p.Wo % 4 == 0 && ((uintptr_t)dst) % (4 * esize) == 0;
    p.dW4 = dw_div(std::max(1, p.W4)); p.dWs = dw_div(p.Ws); p.dRow = dw_div(p.vec_s ? p.Hs * p.W4 : p.Hs * p.Ws); p.dO4 = dw_div(p.Ho * p.O4);
    return true;
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
    Dw3Params q;
    if (dw3_params(g, q, src, dst, (int)sizeof(T), ig)) {
        // about two quads per thread, fewer planes per CTA when that would leave SMs idle
        q.G = std::max(1, std::min(256 / (q.Ho * q.O4), q.planes / (4 * sm_count())));
        while (q.G > 1 && (size_t)q.G * (q.PH * q.PW + 9) * 4 > 48 * 1024 - 16) q.G--;
        const size_t smem = (size_t)q.G * (q.PH * q.PW + 9) * 4;
        const int grid = ceil_div(q.planes, q.G);
        if (smem <= 48 * 1024) {
            if (q.padL == 1) TL_LAUNCH((dw3_kernel<T, 1>), grid, 128, smem, q, src, w, dst);
            else if (q.padL == 0) TL_LAUNCH((dw3_kernel<T, 0>), grid, 128, smem, q, src, w, dst);
            else TL_LAUNCH((dw3_kernel<T, 2>), grid, 128, smem, q, src, w, dst);
            return true;
        }
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
    Dw3Params q;
    if (dw3_params(g, q, x, dy, (int)sizeof(T), false)) {
        groups = std::max(1, std::min(ceil_div(8 * sm_count(), g.Cin), g.n));
        if (dry) return true;
        // all planes of a CTA at once while eight CTAs fit an SM's shared memory: one wait for memory instead of one per plane
        q.G = ceil_div(g.n, groups);
        while (q.G > 1 && (size_t)q.G * q.PH * q.PW * 4 > 24 * 1024) q.G--;
        const size_t smem = (size_t)q.G * q.PH * q.PW * 4;
        const dim3 grid(g.Cin, groups);
#define TL_DW(PADL)                                                                \
    do {                                                                           \
        dw_allow(dw3_wg_kernel<T, PADL>, smem);                                    \
        TL_LAUNCH((dw3_wg_kernel<T, PADL>), grid, 128, smem, q, x, dy, part, g.n); \
    } while (0)
        if (q.padL == 1) TL_DW(1); else if (q.padL == 0) TL_DW(0); else TL_DW(2);
#undef TL_DW
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

// Depthwise convolution, one filter per channel [ref: lib/sources/pulp_conv_naive_fp32.c:29,113,153], for planes that fit
// shared memory.  The layer is bound by memory: nine multiply-adds per value read.  A CTA stages whole planes of one or more
// (stream, channel) pairs with their zero border once (coalesced, each value read once from HBM), and every window is then
// read from shared memory without bounds checks.  64 channels of 28 x 28 x 64 streams, fp32 (25.7 MB per pass): forward 45 us
// and input gradient 92 us with one bounds-checked global read per tap; 145 us for the weight gradient, which ran one CTA per
// (channel, tap).
#include "tl_kernels.h"
#include "tl_reduce.cuh"
#include <algorithm>

namespace tl {

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
    extern __shared__ float dw_smem[];
    const int KH = K ? K : p.Hk, KW = K ? K : p.Wk, KK = KH * KW;
    const int pl0 = blockIdx.x * p.G, np = min(p.G, p.planes - pl0), P = p.PH * p.PW, O = p.Ho * p.Wo;
    float *win = dw_smem, *ws = dw_smem + p.G * P;
    const T *s0 = src + (long long)pl0 * p.Hs * p.Ws;
#pragma unroll 4
    for (int e = threadIdx.x; e < np * P; e += 256) {
        const int g = dw_quot(e, p.dP), rc = e - g * P, r = dw_quot(rc, p.dPW), c = rc - r * p.PW;
        const int h = r + p.r0, x = c + p.c0;
        win[e] = ((unsigned)h < (unsigned)p.Hs && (unsigned)x < (unsigned)p.Ws) ? ld(s0 + (g * p.Hs + h) * p.Ws + x) : 0.f;
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
            dw_smem[e] = ((unsigned)h < (unsigned)p.Hs && (unsigned)xx < (unsigned)p.Ws) ? ld(x + (((long long)(s + g) * p.C + ch) * p.Hs + h) * p.Ws + xx) : 0.f;
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
    DwParams p;
    if (!dw_window(g, p, ig)) return false;
    const int P = p.PH * p.PW, O = p.Ho * p.Wo, KK = g.Hk * g.Wk;
    // about a thousand results per CTA (four per thread), fewer when that would leave SMs idle
    p.G = std::max(1, std::min(1024 / O, p.planes / (2 * sm_count())));
    while (p.G > 1 && (size_t)p.G * (P + KK) * 4 > 48 * 1024) p.G--;
    const size_t smem = (size_t)p.G * (P + KK) * 4;
    const int grid = ceil_div(p.planes, p.G);
#define TL_DW(KV)                                                                                                                   \
    do {                                                                                                                            \
        if (smem > 48 * 1024) cudaFuncSetAttribute(dw_plane_kernel<T, KV>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
        TL_LAUNCH((dw_plane_kernel<T, KV>), grid, 256, smem, p, src, w, dst);                                                       \
    } while (0)
    if (g.Hk == 3 && g.Wk == 3) TL_DW(3); else if (g.Hk == 5 && g.Wk == 5) TL_DW(5); else TL_DW(0);
#undef TL_DW
    return true;
}
// partial weight gradients [groups][C][K*K]; 3 x 3 and 5 x 5 filters.  dry: only the number of groups
template <class T> bool dw_wg_planes(const ConvGeom &g, const T *x, const T *dy, float *part, int &groups, bool dry)
{
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
#define TL_DW(KV)                                                                                                                      \
    do {                                                                                                                               \
        if (smem > 48 * 1024) cudaFuncSetAttribute(dw_wg_plane_kernel<T, KV>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
        TL_LAUNCH((dw_wg_plane_kernel<T, KV>), grid, 256, smem, p, x, dy, part, g.n);                                                  \
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

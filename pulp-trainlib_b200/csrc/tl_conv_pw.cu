// Single-precision pointwise layers (1 x 1, stride 1) over many pixels as 3xTF32 products on tcgen05, each direction in one launch: forward and input
// gradient
//     dst[s][m][p] = sum over k of w[m][k] * src[s][k][p] (+ bias[m])          (input gradient: w transposed)
// [ref: lib/sources/pulp_conv_pw_fp32.c:27 (FW), :233 (IG)]
//
// A product of the GEMM in tl_gemm_tma.cu needs its fp32 operands as packed (hi, lo) copies: three times the activations' bytes written
// and read again, and a launch of its own.  Here the split happens on the way into shared memory.  The pixels of all streams are one
// line of rows, of which each CTA takes one stretch (equal shares: no last wave), 128 rows of D at a time:
//   20 converter warps: four at a time read a piece of 32 channels x 128 pixels (lanes along the pixels, 32 loads a lane in flight), five
//      pieces at once, split it and store it as [hi, lo][4 channels][pixel][16 bytes], which is the tensor core's K-major layout without swizzle;
//   one warp issues D_hi += A_hi B_hi, D_lo += A_hi B_lo + A_lo B_hi (the weights lie behind each other, so that A_hi takes one instruction);
//   four warps add the two parts and store: a lane has a pixel, so a warp stores 32 neighbouring ones of a channel.
// The weights are split once per CTA and stay.  What bounds it: the activations' bytes, from L2 or HBM; figures at pw_covers.
// Every wait is bounded and reports through the status word.
#include "tl_kernels.h"
#include "tl_tc.cuh"
#include <algorithm>

namespace tl {

int *tc_status_word();          // tl_conv_tc.cu

static constexpr int PW_STAGES = 5, PW_CONV = PW_STAGES * 128, PW_THREADS = PW_CONV + 160, PW_KC = 32, PW_MAX_SOURCES = 512;
static constexpr uint32_t PW_HALF = PW_KC / 4 * 128 * 16, PW_STAGE = 2 * PW_HALF, PW_SMEM = 225 * 1024;

struct PwParams {
    const float *src, *w, *bias; float *dst; int *status;
    int P, C, Cd, wm, wk;                       // plane, source and result channels; weight index = m * wm + k * wk
    int total, per;                             // pixels of all streams, of a CTA
    int N, kc, chunks, kpad, stages, accs, cols; // result channels padded; channels of a piece, pieces, channels padded; sets of accumulators
    int chain, chains;                          // pieces that share an accumulator, accumulators of a set (pairs of hi and lo)
};

__device__ __forceinline__ void pw_sts(uint32_t to, const uint32_t *x) { asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(to), "r"(x[0]), "r"(x[1]), "r"(x[2]), "r"(x[3]) : "memory"); }

// CHAINS: several accumulators for the source channels (pw_chains).  Layers with one have a kernel without the loop over them: 1.1 us less for the two
// directions of 64 streams of 64 -> 128 on 28 x 28.
template <bool CHAINS> __global__ void __launch_bounds__(PW_THREADS, 1) conv_pw_kernel(const __grid_constant__ PwParams p)
{
    extern __shared__ __align__(1024) unsigned char pw_smem[];
    __shared__ __align__(8) uint64_t full[PW_STAGES], empty[PW_STAGES], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_s;
    __shared__ int abort_s;
    __shared__ float bias_s[256];
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int lo = blockIdx.x * p.per, hi = min(p.total, lo + p.per), tiles = (hi - lo + 127) / 128, N = p.N, P = p.P, stages = p.stages;
    volatile int *abort_flag = &abort_s;
    const uint32_t a_sm = tc::smem_u32(pw_smem), b_sm = a_sm + (uint32_t)stages * PW_STAGE, b_lbo = (uint32_t)(2 * N + 1) * 16u;
    if (warp == 0) { tc::tmem_alloc(&tmem_s, (uint32_t)p.cols); tc::tmem_relinquish(); }
    if (tid == 32) {
        for (int i = 0; i < stages; i++) { tc::mbar_init(&full[i], 4); tc::mbar_init(&empty[i], 1); }
        for (int i = 0; i < 2; i++) { tc::mbar_init(&acc_full[i], 1); tc::mbar_init(&acc_empty[i], 4); }
        tc::fence_barrier_init();
        abort_s = 0;
    }
    pdl_wait();

    // ---- the first pieces of pixels are on their way while the weights are laid out
    float v[PW_KC];
    const int px = tid & 127, group = warp >> 2, items = tiles * p.chunks;
    int g = lo + px, s = g / P, pp = g - s * P, chunk = group;
    auto wrap = [&] {
        while (chunk >= p.chunks) { chunk -= p.chunks; g += 128; pp += 128; while (pp >= P) { pp -= P; s++; } }
    };
    auto load = [&] {
        const int k = chunk * p.kc, left = g < hi ? min(p.C - k, p.kc) : 0;
        const float *f = p.src + ((long long)s * p.C + k) * P + pp;
        if (left == PW_KC) {
#pragma unroll
            for (int j = 0; j < PW_KC; j++, f += P) v[j] = *f;
        } else {
#pragma unroll
            for (int j = 0; j < PW_KC; j++, f += P) v[j] = j < left ? *f : 0.f;
        }
    };
    wrap();
    if (warp < PW_CONV / 32 && group < stages && group < items) load();
    {
        // neighbouring lanes along the index that is contiguous in memory: 16-byte pieces of four k, rows hi then lo, groups of k an odd
        // number of pieces apart, so that both orders store to all banks
        const int kg = p.kpad / 4, pieces = kg * N;
        const bool k_fast = p.wk == 1;
        for (int e = tid; e < pieces; e += PW_THREADS) {
            const int m = k_fast ? e / kg : e % N, c = k_fast ? e % kg : e / N;
            uint32_t h[4], l[4];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int k = c * 4 + j;
                tc::split_tf32_rn(m < p.Cd && k < p.C ? p.w[(long long)m * p.wm + (long long)k * p.wk] : 0.f, h[j], l[j]);
            }
            pw_sts(b_sm + (uint32_t)c * b_lbo + (uint32_t)m * 16u, h);
            pw_sts(b_sm + (uint32_t)c * b_lbo + (uint32_t)(N + m) * 16u, l);
        }
        if (tid < N) bias_s[tid] = p.bias && tid < p.Cd ? p.bias[tid] : 0.f;
    }
    tc::fence_proxy_async();
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tmem = tmem_s;

    if (warp < PW_CONV / 32) {
        // ---- converters: each group of four warps has a stage of its own (that of every `stages`th piece), so that the stage's
        // barrier is never more than one phase away from what the group waits for
        uint32_t ph = 1;
        for (int i = group; group < stages && i < items; i += stages, ph ^= 1) {
            if (i != group) load();
            if (!tc::warp_wait_or_abort(&empty[group], ph, abort_flag, p.status, 55, 20u, lane)) break;
            const uint32_t to = a_sm + (uint32_t)group * PW_STAGE + (uint32_t)px * 16u;
#pragma unroll
            for (int c = 0; c < PW_KC / 4; c++) {
                if (c % 2 == 0 && c * 4 >= p.kc) break;
                uint32_t h[4], l[4];
#pragma unroll
                for (int j = 0; j < 4; j++) tc::split_tf32_rn(v[c * 4 + j], h[j], l[j]);
                pw_sts(to + (uint32_t)c * 2048u, h);
                pw_sts(to + PW_HALF + (uint32_t)c * 2048u, l);
            }
            tc::fence_proxy_async();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&full[group]);
            chunk += stages;
            wrap();
        }
    } else if (warp == PW_CONV / 32) {
        // ---- the products
        const uint64_t da = tc::smem_desc_kmajor(0u, 2048u, 128u), db = tc::smem_desc_kmajor(0u, b_lbo, 128u);
        const uint32_t a_hw = (uint32_t)(da >> 32), b_hw = (uint32_t)(db >> 32), a_lw0 = (uint32_t)da + (a_sm >> 4), b_lw0 = (uint32_t)db + (b_sm >> 4);
        const bool both = N <= 128;
        const uint32_t id1 = tc::mma_idesc(tc::FMT_TF32, 128, (uint32_t)N), id2 = both ? tc::mma_idesc(tc::FMT_TF32, 128, (uint32_t)(2 * N)) : id1;
        int st = 0; uint32_t ph = 0;
        bool ok = true;
        for (int t = 0; t < tiles && ok; t++) {
            const int buf = p.accs == 2 ? t & 1 : 0, use = p.accs == 2 ? t >> 1 : t;
            if (use && !tc::warp_wait_or_abort(&acc_empty[buf], (uint32_t)(use - 1) & 1u, abort_flag, p.status, 56, 20u, lane)) break;
            tc::tc_fence_after();
            uint32_t d = tmem + (uint32_t)(buf * (CHAINS ? p.chains : 1) * 2 * N), dl = d + (uint32_t)N, bw = b_lw0;
            int first = 0;                                                 // piece with which the chain begins
            for (int c = 0; c < p.chunks; c++) {
                if (CHAINS && c - first == p.chain) { first = c; d += (uint32_t)(2 * N); dl += (uint32_t)(2 * N); }
                if (!tc::warp_wait_or_abort(&full[st], ph, abort_flag, p.status, 57, 0u, lane)) { ok = false; break; }
                tc::tc_fence_after();
                uint32_t aw = a_lw0 + (uint32_t)st * (PW_STAGE / 16);
                const int ks = min(p.kc, p.kpad - c * p.kc) / 8;
                for (int k = 0; k < ks; k++, aw += 256u, bw += 2u * (b_lbo / 16)) {
                    const uint64_t ah = ((uint64_t)a_hw << 32) | aw, al = ((uint64_t)a_hw << 32) | (aw + PW_HALF / 16), bh = ((uint64_t)b_hw << 32) | bw;
                    const uint32_t more = c > first || k > 0;
                    if (tc::elect_one()) {
                        tc::mma_tf32_ss(d, ah, bh, id2, more);
                        if (!both) tc::mma_tf32_ss(dl, ah, ((uint64_t)b_hw << 32) | (bw + (uint32_t)N), id1, more);
                        tc::mma_tf32_ss(dl, al, bh, id1, 1u);
                    }
                }
                if (tc::elect_one()) tc::mma_commit(&empty[st]);
                __syncwarp();
                if (++st == stages) { st = 0; ph ^= 1; }
            }
            if (!ok) break;
            if (tc::elect_one()) tc::mma_commit(&acc_full[buf]);
            __syncwarp();
        }
    } else {
        // ---- results
        const int quad = warp & 3;
        int x = lo + quad * 32 + lane, so = x / P, po = x - so * P;
        for (int t = 0; t < tiles; t++) {
            const int buf = p.accs == 2 ? t & 1 : 0, use = p.accs == 2 ? t >> 1 : t;
            if (!tc::warp_wait_or_abort(&acc_full[buf], (uint32_t)use & 1u, abort_flag, p.status, 58, 20u, lane)) break;
            tc::tc_fence_after();
            const uint32_t d = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(buf * (CHAINS ? p.chains : 1) * 2 * N);
            float *to = p.dst + (long long)so * p.Cd * P + po;
            const bool live = x < hi;
            for (int m = 0; m < N; m += 16) {
                uint32_t a[16], b[16];
                float v[16];
                tc::tmem_ld16(d + (uint32_t)m, a);
                tc::tmem_ld16(d + (uint32_t)(N + m), b);
                tc::tmem_wait_ld();
#pragma unroll
                for (int j = 0; j < 16; j++) v[j] = __uint_as_float(a[j]) + __uint_as_float(b[j]);
                for (int q = 1; CHAINS && q < p.chains; q++) {
                    tc::tmem_ld16(d + (uint32_t)(q * 2 * N + m), a);
                    tc::tmem_ld16(d + (uint32_t)(q * 2 * N + N + m), b);
                    tc::tmem_wait_ld();
#pragma unroll
                    for (int j = 0; j < 16; j++) v[j] += __uint_as_float(a[j]) + __uint_as_float(b[j]);
                }
                if (m + 16 >= N) {                                          // read: the next tile's products may start
                    tc::tc_fence_before();
                    __syncwarp();
                    if (lane == 0) tc::mbar_arrive(&acc_empty[buf]);
                }
                float *y = to + (long long)m * P;
                if (live && m + 16 <= p.Cd) {
#pragma unroll
                    for (int j = 0; j < 16; j++, y += P) *y = v[j] + bias_s[m + j];
                } else if (live) {
#pragma unroll
                    for (int j = 0; j < 16; j++, y += P)
                        if (m + j < p.Cd) *y = v[j] + bias_s[m + j];
                }
            }
            x += 128; po += 128;
            while (po >= P) { po -= P; so++; }
        }
    }
    tc::tc_fence_before();
    __syncthreads();
    if (warp == 0) { tc::tc_fence_after(); tc::tmem_dealloc(tmem, (uint32_t)p.cols); }
}

// The tensor core truncates what it accumulates, so that a chain of steps is as long as those of the kernel that would take the layer
// otherwise.  gemm: one chain, as there (the errors against 64 bits are equal to three digits, 1.69e-6 in both at 300 channels of one sign).
// Else mma.sync, whose chains are at most 16 steps, most of them shorter: two pieces (eight steps), where tensor memory has no
// room for so many accumulators three, and the storing warps add the sums with ordinary rounding.  The error against 64 bits, 30 streams on
// 20 x 20, in units of 1e-7, mma.sync / one chain / here: normal 96 -> 32 3.6 / 2.7 / 1.8, 256 -> 32 4.7 / 6.4 / 2.0, 400 -> 16 4.1 / 9.7 / 2.0, 420 -> 48 7.8 /
// 10.4 / 2.6; terms of one sign 3.6 / 4.3 / 2.3, 4.8 / 14.0 / 2.7, 4.2 / 23.0 / 2.7, 8.9 / 24.4 / 4.0.  From some 500 channels on mma.sync loads its weights
// piece by piece, in chains as short as those (620 -> 32: 2.2 and 1.7; one chain 15 and 38), and takes the layers.
static bool pw_chains(PwParams &p, bool gemm)
{
    p.chain = p.chunks; p.chains = 1;
    if (gemm) return true;
    if (p.C > PW_MAX_SOURCES) return false;
    for (p.chain = 2; p.chain <= 3; p.chain++) {
        p.chains = ceil_div(p.chunks, p.chain);
        if (2 * p.N * p.chains <= 512) return true;
    }
    return false;
}

static bool pw_run(const ConvGeom &g, const float *src, const float *w, const float *bias, float *dst, bool ig)
{
    PwParams p = {};
    p.P = g.Hin * g.Win; p.C = ig ? g.Cout : g.Cin; p.Cd = ig ? g.Cin : g.Cout;
    const long long total = (long long)g.n * p.P;
    if (total >= (1ll << 30) || p.Cd > 256) return false;
    p.kpad = ceil_div(p.C, 8) * 8; p.N = ceil_div(p.Cd, 16) * 16;
    p.chunks = ceil_div(p.kpad, PW_KC); p.kc = ceil_div(ceil_div(p.kpad, p.chunks), 8) * 8;
    p.chunks = ceil_div(p.kpad, p.kc);
    const size_t weights = (size_t)(p.kpad / 4) * (2 * p.N + 1) * 16;
    if (weights + 2 * PW_STAGE > PW_SMEM) return false;
    p.stages = (int)std::min<size_t>(PW_STAGES, (PW_SMEM - weights) / PW_STAGE);
    p.status = tc_status_word();
    if (!p.status) return false;
    if (!pw_chains(p, p.P >= 128 && p.Cd >= 64 && total * p.C * p.Cd >= (1ll << 26))) return false;
    p.accs = 4 * p.N * p.chains <= 512 ? 2 : 1;
    p.cols = 32;
    while (p.cols < 2 * p.N * p.chains * p.accs) p.cols *= 2;
    p.src = src; p.w = w; p.bias = bias; p.dst = dst;
    p.wm = ig ? 1 : g.Cin; p.wk = ig ? g.Cin : 1;
    p.total = (int)total;
    p.per = ceil_div(ceil_div(total, sm_count()), 32) * 32;
    static bool attr = false;
    if (!attr) {
        cudaFuncSetAttribute(conv_pw_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PW_SMEM);
        cudaFuncSetAttribute(conv_pw_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PW_SMEM);
        attr = true;
    }
    const size_t smem = weights + (size_t)p.stages * PW_STAGE;
    if (p.chains > 1) TL_LAUNCH(conv_pw_kernel<true>, ceil_div(total, p.per), PW_THREADS, smem, p);
    else TL_LAUNCH(conv_pw_kernel<false>, ceil_div(total, p.per), PW_THREADS, smem, p);
    profile_add_flops(2.0 * total * g.Cin * g.Cout);
    return true;
}

// Where it pays.  Every CTA splits all weights, so that it takes pixels to spread: below 64 for each SM the layers stay on mma.sync, whose
// shorter accumulation chains there (few tiles, split sums) are also the more exact ones, or on the GEMM.  Measured over eighty random layers
// (us, before / here; "GEMM": packed operands, "mma": mma.sync; the error against 64 bits is the GEMM's to three digits and a third to all of mma.sync's):
//   64 streams of 64 -> 128 on 28 x 28: GEMM 23.0 / 11.8 forward, 24.4 / 12.6 back;  512 of 64 -> 64 on 32 x 32: 131 / 53 (5.1 TB/s)
//   16 of 64 -> 128 on 28 x 28: 10.2 / 7.2;  8 of 96 -> 120 on 30 x 30 (7200 pixels) 11.5 / 8.7;  2 of 64 -> 256 on 48 x 48 (4608) 9.5 / 10.1
//   128 of 64 -> 32 on 40 x 40: mma 38 / 15;  a layer of 21840 pixels, 56 -> 66 on 7 x 13: 22.1 / 7.9;  of 12920, 22 -> 129 on 17 x 19: 15.1 / 6.0
//   few channels on even planes, which mma.sync stages two pixels at a time: 30600 pixels of 4 -> 7 4.4 / 4.7, 28160 of 16 -> 8 4.7 / 4.9,
//     83356 of 2 -> 13 10.0 / 7.4
//   fewer pixels: 2400 of 52 -> 66 8.5 / 6.2, but with twice the error; 540 of 7 -> 90 4.1 / 4.8
static bool pw_covers(const ConvGeom &g, int sources, int results)
{
    if (g.depthwise || gemm_path() != 0 || g.Hk != 1 || g.Wk != 1 || g.sh != 1 || g.sw != 1 || g.padU != 0 || g.padL != 0 || g.Hin != g.Hout || g.Win != g.Wout) return false;
    const long long P = (long long)g.Hin * g.Win, total = g.n * P;
    if (total < 64ll * sm_count()) return g.n > 1 && P >= 128 && results >= 64 && total >= 48ll * sm_count() && total * sources * results >= (1ll << 26);     // the GEMM's layers
    return P >= 16 && (std::max(sources, results) > 16 || total * (sources + results) >= 700000);
}
// false = not covered, nothing launched
bool conv_pw_fw(const ConvGeom &g, const float *x, const float *w, const float *bias, float *y) { return pw_covers(g, g.Cin, g.Cout) && pw_run(g, x, w, bias, y, false); }
bool conv_pw_ig(const ConvGeom &g, const float *dy, const float *w, float *dx) { return pw_covers(g, g.Cout, g.Cin) && pw_run(g, dy, w, nullptr, dx, true); }

// ---------------------------------------------------------------- weight gradient
//     dW[co][ci] = sum over the pixels of all streams of dY[co][p] * X[ci][p]          [ref: lib/sources/pulp_conv_pw_fp32.c:121]
// The contraction runs over the pixels, which are contiguous in memory: four of them are a 16-byte piece of the K-major layout as they
// come.  A CTA takes one stretch of the pixels, 32 at a time (three groups of four converter warps, each with a stage of its own): rows of
// X in hi and lo, rows of dY in hi and lo.  The tensor core truncates what it accumulates, so a chain is four k-steps long: each piece has a
// fresh accumulator (two banks), and eight warps add it to sums that they hold in registers.  Lanes are source channels, so that a
// CTA's partial result is written coalesced in the layout of dW; a second launch adds the partial results.
static constexpr int PWW_GROUPS = 3, PWW_STAGES = 2 * PWW_GROUPS, PWW_CONV = PWW_GROUPS * 128, PWW_ISSUERS = 2, PWW_THREADS = PWW_CONV + PWW_ISSUERS * 32 + 256;

struct PwWgParams {
    const float *x, *dy; float *part; int *status;
    int P, Cin, Cout, total, per;               // plane, channels, pixels of all streams, of a CTA
    int N, co_slices, RA, la, fold, lbo, cols;  // result channels of a slice, slices of them; source channels of a slice, padded; rows to their lo parts; pieces of four pixels
    uint32_t stage_bytes;
};

// Rows u = 0, 1, ... of a lane, a step apart: of X up to nx, of dY from there to nu (the same in all lanes of a warp); `have`: those that exist.
template <bool VEC> __device__ __forceinline__ void pw_wg_load(const float *f, const float *fy, long long step, float (&v)[8][4], int nx, int nu, uint32_t have,
                                                               int left, int wrap, long long next_x, long long next_y)
{
#pragma unroll
    for (int u = 0; u < 8; u++, f += step) {
        if (u >= nu) break;
        if (u == nx) f = fy;
        const bool ok = (have >> u) & 1;
        if (VEC) {
            float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
            if (ok) q = *reinterpret_cast<const float4 *>(f);
            v[u][0] = q.x; v[u][1] = q.y; v[u][2] = q.z; v[u][3] = q.w;
        } else {
            const long long next = u < nx ? next_x : next_y;                                   // from the end of a plane to the next stream's
#pragma unroll
            for (int e = 0; e < 4; e++) v[u][e] = ok && e < left ? f[e + (e >= wrap ? next : 0)] : 0.f;
        }
    }
}
__device__ __forceinline__ void pw_wg_store(const float (&v)[8][4], uint32_t to, uint32_t to_y, uint32_t lo_x, uint32_t lo_y, uint32_t step, int nx, int nu)
{
#pragma unroll
    for (int u = 0; u < 8; u++) {
        if (u >= nu) break;
        uint32_t h[4], l[4];
#pragma unroll
        for (int e = 0; e < 4; e++) tc::split_tf32_rn(v[u][e], h[e], l[e]);
        const uint32_t at = (u < nx ? to : to_y) + (uint32_t)u * step;
        pw_sts(at, h);
        pw_sts(at + (u < nx ? lo_x : lo_y), l);
    }
}

template <bool VEC, int PX> __global__ void __launch_bounds__(PWW_THREADS, 1) conv_pw_wg_kernel(const __grid_constant__ PwWgParams p)
{
    constexpr int KG = PX / 4, RS = 128 / KG, IB = 32 / PX;                 // pieces of four pixels, rows that a group of warps loads at once, pieces of an accumulator
    extern __shared__ __align__(1024) unsigned char pw_smem[];
    __shared__ __align__(8) uint64_t full[PWW_STAGES], empty[PWW_STAGES], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_s;
    __shared__ int abort_s;
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int lo = blockIdx.x * p.per, hi = min(p.total, lo + p.per), pieces = (hi - lo + PX - 1) / PX, N = p.N, P = p.P;
    const int co0 = ((int)blockIdx.y % p.co_slices) * N, ci0 = ((int)blockIdx.y / p.co_slices) * p.RA;
    volatile int *abort_flag = &abort_s;
    const uint32_t sm = tc::smem_u32(pw_smem);
    if (warp == 0) { tc::tmem_alloc(&tmem_s, (uint32_t)p.cols); tc::tmem_relinquish(); }
    if (tid == 32) {
        for (int i = 0; i < PWW_STAGES; i++) { tc::mbar_init(&full[i], 4); tc::mbar_init(&empty[i], 1); }
        for (int i = 0; i < 2; i++) { tc::mbar_init(&acc_full[i], 1); tc::mbar_init(&acc_empty[i], 8); }
        tc::fence_barrier_init();
        abort_s = 0;
    }
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tmem = tmem_s;
    pdl_wait();

    if (warp < PWW_CONV / 32) {
        const int group = warp >> 2, kg = lane % KG, wq = RS / 4 * (warp & 3), r0 = lane / KG + wq;
        const int nx = (p.RA - wq + RS - 1) / RS, nu = (p.RA + N - wq + RS - 1) / RS;
        uint32_t have = 0;
        for (int u = 0; u < nu; u++) have |= (uint32_t)(u < nx ? ci0 + r0 + RS * u < p.Cin : co0 + r0 + RS * u - p.RA < p.Cout) << u;
        int g = lo + group * PX + kg * 4, s = g / P, pp = g - s * P;
        const float *x = p.x + ((long long)s * p.Cin + ci0 + r0) * P + pp, *y = p.dy + ((long long)s * p.Cout + co0 + r0 + RS * nx - p.RA) * P + pp;
        const long long step = (long long)RS * P, next_x = (long long)(p.Cin - 1) * P, next_y = (long long)(p.Cout - 1) * P;
        const uint32_t to = sm + (uint32_t)group * p.stage_bytes + (uint32_t)(kg * p.lbo + r0) * 16u, lo_x = (uint32_t)p.la * 16u, lo_y = (uint32_t)N * 16u;
        float v[8][4];
        for (int c = group, t = 0; c < pieces; c += PWW_GROUPS, t++) {
            pw_wg_load<VEC>(x, y, step, v, nx, nu, g < hi ? have : 0u, hi - g, P - pp, next_x, next_y);
            const int st = group + (t & 1) * PWW_GROUPS;
            if (!tc::warp_wait_or_abort(&empty[st], (uint32_t)(~t >> 1) & 1u, abort_flag, p.status, 59, 20u, lane)) break;
            const uint32_t at = to + (uint32_t)((t & 1) * PWW_GROUPS) * p.stage_bytes;
            pw_wg_store(v, at, at + (uint32_t)(2 * p.la - p.RA) * 16u, lo_x, lo_y, RS * 16u, nx, nu);
            tc::fence_proxy_async();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&full[st]);
            g += PWW_GROUPS * PX; pp += PWW_GROUPS * PX; x += PWW_GROUPS * PX; y += PWW_GROUPS * PX;
            while (pp >= P) { pp -= P; x += next_x; y += next_y; }
        }
    } else if (warp < PWW_CONV / 32 + PWW_ISSUERS) {
        // ---- the products: 32 pixels for an accumulator, each issuing warp one of the two (a wait, a commit and a product cost one warp 100 to
        // 150 cycles each whatever their size)
        const uint64_t d0 = tc::smem_desc_kmajor(0u, (uint32_t)p.lbo * 16u, 128u);
        const uint32_t hw = (uint32_t)(d0 >> 32), lw0 = (uint32_t)d0 + (sm >> 4);
        const uint32_t id1 = tc::mma_idesc(tc::FMT_TF32, 128, (uint32_t)N), id2 = tc::mma_idesc(tc::FMT_TF32, 128, (uint32_t)(2 * N));
        const int bank = warp - PWW_CONV / 32;
        const uint32_t d = tmem + (uint32_t)(bank * 2 * N);
        int st = IB * bank; uint32_t ph = 0, use = 0;
        bool ok = true;
        for (int c0 = IB * bank; c0 < pieces && ok; c0 += IB * PWW_ISSUERS, use++) {
            if (use && !tc::warp_wait_or_abort(&acc_empty[bank], (use - 1) & 1u, abort_flag, p.status, 60, 0u, lane)) break;
            for (int c = c0; c < min(pieces, c0 + IB); c++, st++) {
                if (!tc::warp_wait_or_abort(&full[st], ph, abort_flag, p.status, 61, 0u, lane)) { ok = false; break; }
                tc::tc_fence_after();
                uint32_t aw = lw0 + (uint32_t)st * (p.stage_bytes / 16);
#pragma unroll
                for (int k = 0; k < PX / 8; k++, aw += 2u * (uint32_t)p.lbo) {
                    const uint64_t ah = ((uint64_t)hw << 32) | aw, al = ah + (uint32_t)p.la, bh = ah + (uint32_t)(2 * p.la);
                    if (tc::elect_one()) {
                        tc::mma_tf32_ss(d, ah, bh, id2, (uint32_t)(c > c0 || k > 0));
                        if (!p.fold) tc::mma_tf32_ss(d + (uint32_t)N, al, bh, id1, 1u);
                    }
                }
                if (tc::elect_one()) tc::mma_commit(&empty[st]);
                __syncwarp();
            }
            if (!ok) break;
            if (tc::elect_one()) tc::mma_commit(&acc_full[bank]);
            __syncwarp();
            st += IB * (PWW_ISSUERS - 1);
            if (st >= PWW_STAGES) { st -= PWW_STAGES; ph ^= 1; }
        }
    } else {
        // ---- sums: a lane has a source channel, each set of four warps half of the result channels
        const int quad = warp & 3, set = (warp - PWW_CONV / 32 - PWW_ISSUERS) >> 2, ng = N / 16, half = (ng + 1) / 2, first = set * half, count = min(half, ng - first);
        float acc[4][16];
#pragma unroll
        for (int q = 0; q < 4; q++)
#pragma unroll
            for (int j = 0; j < 16; j++) acc[q][j] = 0.f;
        bool ok = true;
        for (int c = 0; c < (pieces + IB - 1) / IB; c++) {
            const int bank = c & 1;
            if (!tc::warp_wait_or_abort(&acc_full[bank], (uint32_t)(c >> 1) & 1u, abort_flag, p.status, 62, 20u, lane)) { ok = false; break; }
            tc::tc_fence_after();
            const uint32_t d = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(bank * 2 * N + first * 16);
#pragma unroll
            for (int q = 0; q < 4; q++) {
                if (q < count) {
#pragma unroll
                    for (int e = 0; e < 16; e += 8) {
                        uint32_t a[8], b[8];
                        tc::tmem_ld8(d + (uint32_t)(q * 16 + e), a);
                        tc::tmem_ld8(d + (uint32_t)(N + q * 16 + e), b);
                        tc::tmem_wait_ld();
#pragma unroll
                        for (int j = 0; j < 8; j++) acc[q][e + j] += __uint_as_float(a[j]) + __uint_as_float(b[j]);
                    }
                }
            }
            tc::tc_fence_before();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&acc_empty[bank]);
        }
        const int row = quad * 32 + lane, ci = ci0 + row;
        if (p.fold) {                                                       // the products of X_lo, in lanes 64 .. 127
            float *other = reinterpret_cast<float *>(pw_smem) + (set * 64) * 64 + (row & 63);
            if (row >= 64) {
#pragma unroll
                for (int q = 0; q < 4; q++)
#pragma unroll
                    for (int j = 0; j < 16; j++) other[(q * 16 + j) * 64] = acc[q][j];
            }
            asm volatile("bar.sync 1, 256;" ::: "memory");
            if (row < 64) {
#pragma unroll
                for (int q = 0; q < 4; q++)
#pragma unroll
                    for (int j = 0; j < 16; j++) acc[q][j] += other[(q * 16 + j) * 64];
            }
        }
        if (ok && row < p.RA && ci < p.Cin) {
            float *to = p.part + (long long)blockIdx.x * p.Cin * p.Cout + ci;
#pragma unroll
            for (int q = 0; q < 4; q++)
#pragma unroll
                for (int j = 0; j < 16; j++) {
                    const int co = co0 + (first + q) * 16 + j;
                    if (q < count && co < p.Cout) to[(long long)co * p.Cin] = acc[q][j];
                }
        }
    }
    tc::tc_fence_before();
    __syncthreads();
    if (warp == 0) { tc::tc_fence_after(); tc::tmem_dealloc(tmem, (uint32_t)p.cols); }
}

// One partial result per CTA into `part`, their number into *groups; dry_run: only that; false = not covered.
// What bounds it: the converter warps' chain of load, split, store and hand-over at three pieces in flight (64 -> 64 channels, a piece of 32 pixels:
// 1200 cycles, where its bytes take 650); loading the next piece's first half between the stores of this one was slower (the proxy
// fence waits for loads in flight), 16 pixels at a time took 1.3 times as long for up to 128 rows.  Measured with the sum of the
// partial results over eighty random layers (us, mma.sync / here):
//   64 streams of 64 -> 128 on 28 x 28 32.6 / 19.6;  64 of 160 -> 96 on 20 x 20 58.5 / 17.0;  512 of 64 -> 64 on 32 x 32 130 / 77;  256 of 128 -> 64
//     on 28 x 28 126 / 51;  45402 pixels of 14 -> 24 14.5 / 13.7
// The error against 64 bits is 0.65 to 1.08 times that of mma.sync's (the mean 0.95; shorter sums in registers, from more CTAs, cost
// 3 to 30 us at 200 to 500 thousand pixels and did not change it).
//   few pixels: 7161 of 72 -> 72 14.7 / 11.8, 9976 of 8 -> 95 9.7 / 11.8, 4797 of 6 -> 16 7.6 / 8.5, 2400 of 52 -> 66 10.0 / 10.5
bool conv_pw_wg(const ConvGeom &g, const float *x, const float *dy, float *part, int *groups, bool dry_run)
{
    if (g.depthwise || gemm_path() != 0 || g.Hk != 1 || g.Wk != 1 || g.sh != 1 || g.sw != 1 || g.padU != 0 || g.padL != 0 || g.Hin != g.Hout || g.Win != g.Wout) return false;
    const long long total = (long long)g.n * g.Hin * g.Win;
    if (total >= (1ll << 30) || g.Hin * g.Win < 16) return false;
    if (total < 72ll * sm_count() && !(total >= 48ll * sm_count() && g.Cin >= 32 && g.Cout >= 32)) return false;
    PwWgParams p = {};
    p.P = g.Hin * g.Win; p.Cin = g.Cin; p.Cout = g.Cout; p.total = (int)total;
    p.co_slices = ceil_div(g.Cout, 128);
    p.N = ceil_div(ceil_div(g.Cout, p.co_slices), 16) * 16;
    const int ci_slices = ceil_div(g.Cin, 128), slices = p.co_slices * ci_slices;
    p.RA = ceil_div(ceil_div(g.Cin, ci_slices), 16) * 16;
    if (slices > sm_count() / 8) return false;
    p.fold = p.RA <= 64; p.la = p.fold ? 64 : p.RA;
    const int px = p.RA + p.N <= 128 && PWW_STAGES * 8u * (2 * (p.la + p.N) + 1) * 16 + 2048 <= PW_SMEM ? 32 : 16;      // pixels of a piece: eight 16-byte loads a lane
    p.lbo = 2 * (p.la + p.N) + (px == 32 ? 1 : 2);                         // an odd number: eight groups of pixels store to all banks; two past a multiple of eight: four groups x two rows do
    p.stage_bytes = (uint32_t)(px / 4 * p.lbo) * 16u;
    p.per = std::max(128, ceil_div(ceil_div(total, sm_count() / slices), 32) * 32);
    *groups = ceil_div(total, p.per);
    if (dry_run) return true;
    p.cols = 32;
    while (p.cols < 4 * p.N) p.cols *= 2;
    p.x = x; p.dy = dy; p.part = part; p.status = tc_status_word();
    if (!p.status) return false;
    // the products read 128 rows whatever X has: rows past the last are not used, but have to lie in shared memory
    const size_t smem = PWW_STAGES * (size_t)p.stage_bytes + 128 * 16;
    const bool vec = p.P % 4 == 0 && (((uintptr_t)x | (uintptr_t)dy) & 15) == 0;
    static bool attr = false;
    if (!attr) {
        cudaFuncSetAttribute(conv_pw_wg_kernel<true, 32>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PW_SMEM);
        cudaFuncSetAttribute(conv_pw_wg_kernel<false, 32>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PW_SMEM);
        cudaFuncSetAttribute(conv_pw_wg_kernel<true, 16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PW_SMEM);
        cudaFuncSetAttribute(conv_pw_wg_kernel<false, 16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PW_SMEM);
        attr = true;
    }
    const dim3 grid(*groups, slices);
    if (px == 32 && vec) TL_LAUNCH((conv_pw_wg_kernel<true, 32>), grid, PWW_THREADS, smem, p);
    else if (px == 32) TL_LAUNCH((conv_pw_wg_kernel<false, 32>), grid, PWW_THREADS, smem, p);
    else if (vec) TL_LAUNCH((conv_pw_wg_kernel<true, 16>), grid, PWW_THREADS, smem, p);
    else TL_LAUNCH((conv_pw_wg_kernel<false, 16>), grid, PWW_THREADS, smem, p);
    profile_add_flops(2.0 * total * g.Cin * g.Cout);
    return true;
}

} // namespace tl

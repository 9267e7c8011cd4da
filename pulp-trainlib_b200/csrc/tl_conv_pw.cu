// Single-precision pointwise layers (1 x 1, stride 1) over many pixels in one launch: forward and input gradient as 3xTF32 products on tcgen05
//     dst[s][m][p] = sum over k of w[m][k] * src[s][k][p] (+ bias[m])          (input gradient: w transposed)
// [ref: lib/sources/pulp_conv_pw_fp32.c:27 (FW), :233 (IG)]
//
// A product of the GEMM in tl_gemm_tma.cu needs its fp32 operands as packed (hi, lo) copies: three times the activations' bytes written
// and read again, and a launch of its own.  Here the split happens on the way into shared memory.  The pixels of all streams are one
// line of rows, of which each CTA takes one stretch (equal shares: no last wave), 128 rows of D at a time:
//   20 converter warps read 32 channels x 128 pixels at a time (lanes along the pixels; four warps take a piece of 32 loads a lane, five pieces are in flight), split and
//      store them as [hi, lo][4 channels][pixel][16 bytes], which is the tensor core's K-major layout without swizzle;
//   one warp issues D_hi += A_hi B_hi, D_lo += A_hi B_lo + A_lo B_hi (the weights lie behind each other, so that A_hi takes one instruction);
//   four warps add the two parts and store: a lane has a pixel, so a warp stores 32 neighbouring ones of a channel.
// The weights are split once per CTA and stay.  What bounds it: the activations' bytes, from L2 or HBM; figures at pw_covers.
// Every wait is bounded and reports through the status word.
#include "tl_kernels.h"
#include "tl_tc.cuh"
#include <algorithm>

namespace tl {

int *tc_status_word();          // tl_conv_tc.cu

static constexpr int PW_STAGES = 5, PW_CONV = PW_STAGES * 128, PW_THREADS = PW_CONV + 160, PW_KC = 32;
static constexpr uint32_t PW_HALF = PW_KC / 4 * 128 * 16, PW_STAGE = 2 * PW_HALF, PW_SMEM = 225 * 1024;

struct PwParams {
    const float *src, *w, *bias; float *dst; int *status;
    int P, C, Cd, wm, wk;                       // plane, source and result channels; weight index = m * wm + k * wk
    int total, per;                             // pixels of all streams, of a CTA
    int N, kc, chunks, kpad, stages, accs, cols; // result channels padded; channels of a piece, pieces, channels padded; accumulators
};

__device__ __forceinline__ void pw_split(float x, uint32_t &hi, uint32_t &lo)
{
    tc::split_tf32_fast(x, hi, lo);
    lo += 0x1000u;                              // the tensor core cuts it off
}
__device__ __forceinline__ void pw_sts(uint32_t to, const uint32_t *x) { asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(to), "r"(x[0]), "r"(x[1]), "r"(x[2]), "r"(x[3]) : "memory"); }

__global__ void __launch_bounds__(PW_THREADS, 1) conv_pw_kernel(const __grid_constant__ PwParams p)
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
                pw_split(m < p.Cd && k < p.C ? p.w[(long long)m * p.wm + (long long)k * p.wk] : 0.f, h[j], l[j]);
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
                for (int j = 0; j < 4; j++) pw_split(v[c * 4 + j], h[j], l[j]);
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
            const uint32_t d = tmem + (uint32_t)(buf * 2 * N), dl = d + (uint32_t)N;
            uint32_t bw = b_lw0;
            for (int c = 0; c < p.chunks; c++) {
                if (!tc::warp_wait_or_abort(&full[st], ph, abort_flag, p.status, 57, 0u, lane)) { ok = false; break; }
                tc::tc_fence_after();
                uint32_t aw = a_lw0 + (uint32_t)st * (PW_STAGE / 16);
                const int ks = min(p.kc, p.kpad - c * p.kc) / 8;
                for (int k = 0; k < ks; k++, aw += 256u, bw += 2u * (b_lbo / 16)) {
                    const uint64_t ah = ((uint64_t)a_hw << 32) | aw, al = ((uint64_t)a_hw << 32) | (aw + PW_HALF / 16), bh = ((uint64_t)b_hw << 32) | bw;
                    const uint32_t more = c > 0 || k > 0;
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
            const uint32_t d = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(buf * 2 * N);
            float *to = p.dst + (long long)so * p.Cd * P + po;
            const bool live = x < hi;
            for (int m = 0; m < N; m += 16) {
                uint32_t a[16], b[16];
                tc::tmem_ld16(d + (uint32_t)m, a);
                tc::tmem_ld16(d + (uint32_t)(N + m), b);
                tc::tmem_wait_ld();
                if (m + 16 >= N) {                                          // read: the next tile's products may start
                    tc::tc_fence_before();
                    __syncwarp();
                    if (lane == 0) tc::mbar_arrive(&acc_empty[buf]);
                }
                float *y = to + (long long)m * P;
                if (live && m + 16 <= p.Cd) {
#pragma unroll
                    for (int j = 0; j < 16; j++, y += P) *y = __uint_as_float(a[j]) + __uint_as_float(b[j]) + bias_s[m + j];
                } else if (live) {
#pragma unroll
                    for (int j = 0; j < 16; j++, y += P)
                        if (m + j < p.Cd) *y = __uint_as_float(a[j]) + __uint_as_float(b[j]) + bias_s[m + j];
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
    p.accs = 4 * p.N <= 512 ? 2 : 1;
    p.cols = 32;
    while (p.cols < 2 * p.N * p.accs) p.cols *= 2;
    p.src = src; p.w = w; p.bias = bias; p.dst = dst;
    p.wm = ig ? 1 : g.Cin; p.wk = ig ? g.Cin : 1;
    p.total = (int)total;
    p.per = ceil_div(ceil_div(total, sm_count()), 32) * 32;
    static bool attr = false;
    if (!attr) { cudaFuncSetAttribute(conv_pw_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PW_SMEM); attr = true; }
    TL_LAUNCH(conv_pw_kernel, ceil_div(total, p.per), PW_THREADS, weights + (size_t)p.stages * PW_STAGE, p);
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

} // namespace tl

// Matrix products below the size where the TMA-fed tcgen05 kernels pay (tl_gemm_tma.cu), as one launch for a whole group:
// up to GG_MAX products of different shapes (the three projections of an attention layer, the five gradients behind its
// core), each with any operand strides, a batch, and a contraction that may run over several segments (separate
// allocations, or the streams of a batch).  Replaces the mm / mm_M / mm_unroll_* family at these sizes
// [ref: lib/sources/pulp_matmul_fp32.c:190-3697, pulp_matmul_fp16.c:191-1908].
//
// What bounds these products is not arithmetic but the chain launch -> first operand bytes -> last store: a 256^3 product
// is half a microsecond of FFMA work on 148 SMs.  Hence small tiles (many CTAs), the whole CTA loading a long K chunk with
// asynchronous copies at once, and the K steps of a chunk dealt to the WARPS of the CTA (every warp owns the whole tile for
// its share of K; the partial tiles meet in shared memory in warp order).  Outputs with fewer tiles than SMs are further
// split along K over CTAs; the CTA of a tile that finishes last adds the splits in order, so results do not depend on
// scheduling.  Where a 128 x 128 x 512 product of one chunk spends its 3500 cycles (clock counters, fp16): 1000 in front of the first
// copy (1600 with divisions by variables), 800 issuing copies, 250 waiting, 680 multiplying, 120 exchanging, 600 storing (1050
// with the parameters of the end first read there).
//   fp32: FFMA (full fp32 products and sums), 4 x 4 results per lane, operands read as 16-byte vectors along
//         whichever of k / row is contiguous in memory: no transposition on the way into shared memory.
//   fp16: mma.sync.m16n8k16 with fp32 accumulation, fragments by ldmatrix (plain for K-contiguous operands, .trans for
//         row-contiguous ones).  A tcgen05 tile needs 128 rows and a barrier/TMEM set-up that costs more than these
//         products take.
#include "tl_kernels.h"
#include <algorithm>
#include <type_traits>
#include <cstdlib>

namespace tl {

static constexpr int GG_MAX = 6;

// n / d by multiplication, exact while n d < 2^32; m = 1: by division, where n may be larger than that (a division by a variable costs
// a warp about a hundred cycles, and the chain of them in front of the first copy was a third of a small product's time)
struct GgDiv { uint32_t m; int d; };
static GgDiv gg_div(int d, long long n_max) { GgDiv r; r.d = d; r.m = d == 1 ? 0u : n_max * d < (1ll << 32) ? (uint32_t)(((1ull << 32) + d - 1) / d) : 1u; return r; }
__device__ __forceinline__ int gg_quot(int n, GgDiv d) { return d.m > 1u ? (int)__umulhi((uint32_t)n, d.m) : d.m ? n / d.d : n; }

template <class T> struct GgProb {
    const T *A[3], *B[3]; T *C; const T *bias;
    int N, M, K, segs, seg_list;                // seg_list: segment s uses A[s], B[s]; else A[0] + s * a_ss, B[0] + s * b_ss
    int a_kc, b_kc;                             // 1: k is the contiguous (or nearest) index of the operand, 0: its row
    int a_vl, b_vl;                             // log2 of the elements per copy (16 bytes, 4 bytes or one element)
    GgDiv tiles_m, tiles_nm, splits;            // column tiles, tiles per matrix, CTAs per tile
    GgDiv cps;                                  // K chunks of a segment
    int chunks, per;                            // K chunks in all, of one CTA
    int quads, plain;                           // four neighbouring results may be stored at once / and nothing is added to them
    long long a_cs, a_ss_, b_cs, b_ss_;         // strides of the contiguous-side and the other index (a_cs: usually 1)
    long long a_bs, b_bs, c_bs, a_ks, b_ks;     // batch strides, segment strides
    long long c_rs, c_cs;
    float alpha; int accumulate, bias_mode, ticket0;
    float *part;                                // [tile][split][BM * BN]
};
// G: room for so many products (a launch of one product has its parameters at fixed addresses); first: the first CTA of each (past the grid: none)
template <class T, int G> struct GgParams { int first[G]; GgProb<T> p[G]; };

static __device__ unsigned gg_tickets[16384];   // one per tile of a K-split product; zero between launches

__device__ __forceinline__ void gg_cp16(uint32_t dst, const void *src, int bytes)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void gg_cp4(uint32_t dst, const void *src, int bytes)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

// Copies of one operand's tiles into shared memory as [TS strided][TC contiguous + PAD] (K-contiguous operands: TC = KC,
// TS = rows; row-contiguous ones the other way round).  Both layouts move the same number of pieces per thread and chunk, so
// one loop serves both: everything that depends on the layout, the strides and the thread is worked out once per tile, a
// piece then costs a compare, an address add and the copy.  Elements outside the matrix become zero.
template <class T, int ROWS, int KC, int PAD, int NT> struct GgLoader {
    static constexpr int SZ = (int)sizeof(T), V16 = 16 / SZ, V4 = 4 / SZ;
    const char *ptr, *safe;     // this thread's first element of the current chunk / any valid address
    long long pass, chunk;      // bytes from one piece of the thread to the next, from one chunk to the next
    uint32_t sm, sm_pass;       // byte offset of the first piece in the stage, step
    int s, s_step, c, kc, vw, lim_c, lim_s;    // strided / contiguous index of the first piece; limits of the non-k index

    static constexpr int log2c(int n) { return n <= 1 ? 0 : 1 + log2c(n / 2); }
    __device__ __forceinline__ void init(const T *src, int kc_, int vl, int row0, int k0, int rows, long long cs, long long ss)
    {
        kc = kc_; vw = 1 << vl;
        const int tc = kc ? KC : ROWS, pl = (kc ? log2c(KC) : log2c(ROWS)) - vl;       // pieces per shared-memory row: powers of two
        const int tid = threadIdx.x;
        s = tid >> pl; c = (tid & ((1 << pl) - 1)) << vl; s_step = NT >> pl;
        const int pitch = tc + PAD;
        sm = (uint32_t)((s * pitch + c) * SZ); sm_pass = (uint32_t)(s_step * pitch * SZ);
        const long long c0 = kc ? k0 : row0, s0 = kc ? row0 : k0;
        safe = reinterpret_cast<const char *>(src);
        ptr = safe + ((s0 + s) * ss + (c0 + c) * cs) * SZ;
        pass = (long long)s_step * ss * SZ; chunk = (kc ? (long long)KC * cs : (long long)KC * ss) * SZ;
        lim_c = rows - row0; lim_s = rows - row0;
    }
    // k_left: rows of k from this chunk's start to the end of the segment
    __device__ __forceinline__ void fetch(uint32_t stage, int k_left)
    {
        const int ls = kc ? lim_s : k_left, lc = (kc ? k_left : lim_c) - c;
        if (vw == V16) {
            const int cb = min(max(lc, 0), V16) * SZ;
            constexpr int Q = ROWS * KC / V16 / NT;
#pragma unroll
            for (int q = 0; q < Q; q++) {
                const int b = s + q * s_step < ls ? cb : 0;
                gg_cp16(stage + sm + q * sm_pass, b ? ptr + q * pass : safe, b);
            }
        } else if (SZ == 4 || vw == V4) {
            const int cb = min(max(lc, 0), V4) * SZ;
            constexpr int Q = ROWS * KC / V4 / NT;
            const char *from = ptr;
            uint32_t to = stage + sm;
            if (__all_sync(0xffffffffu, s + (Q - 1) * s_step < ls && lc >= V4)) {
                // all of a warp's pieces inside the matrix: half the instructions of a piece are its limits
#pragma unroll 8
                for (int q = 0; q < Q; q++, from += pass, to += sm_pass) gg_cp4(to, from, 4);
            } else {
#pragma unroll 8
                for (int q = 0; q < Q; q++, from += pass, to += sm_pass) {
                    const int b = s + q * s_step < ls ? cb : 0;
                    gg_cp4(to, b ? from : safe, b);
                }
            }
        } else {
            constexpr int Q = ROWS * KC / NT, U = 8;
            for (int q0 = 0; q0 < Q; q0 += U) {
                unsigned short v[U];
#pragma unroll
                for (int u = 0; u < U; u++) v[u] = (s + (q0 + u) * s_step < ls && lc > 0) ? *reinterpret_cast<const unsigned short *>(ptr + (q0 + u) * pass) : (unsigned short)0;
#pragma unroll
                for (int u = 0; u < U; u++) asm volatile("st.shared.u16 [%0], %1;" ::"r"(stage + sm + (q0 + u) * sm_pass), "h"(v[u]) : "memory");
            }
        }
        ptr += chunk;
    }
};

// ---------------------------------------------------------------- the share of one warp in one K chunk
// fp32: lanes are 4 x 8; a lane owns RM x RN results.  Rows of a K-contiguous operand are dealt round-robin to the lanes
// (row = lane row + 4 r: neighbouring lanes read neighbouring shared-memory rows, 4 banks apart), rows of a row-contiguous
// one in quads (one 16-byte read per k).  The results of a lane follow the same maps (gg_row / gg_col).
template <int RM> __device__ __forceinline__ int gg_row(int r, int lr, int kc) { return kc ? lr + 4 * r : (r / 4) * 16 + lr * 4 + (r & 3); }
template <int RN> __device__ __forceinline__ int gg_col(int c, int lc, int kc) { return kc ? lc + 8 * c : (c / 4) * 32 + lc * 4 + (c & 3); }

template <bool a_kc, bool b_kc, int RM, int RN, int PA_K, int PA_R, int PB_K, int PB_R, int KW>
__device__ __forceinline__ void gg_ffma(const float *As, const float *Bs, int k0, float (&acc)[RM][RN], int lr, int lc)
{
#pragma unroll 2
    for (int k = k0; k < k0 + KW; k += 4) {
        float a[RM][4], b[RN][4];
        if (a_kc) {
#pragma unroll
            for (int r = 0; r < RM; r++) { const float4 v = *reinterpret_cast<const float4 *>(As + (lr + 4 * r) * PA_K + k); a[r][0] = v.x; a[r][1] = v.y; a[r][2] = v.z; a[r][3] = v.w; }
        } else {
#pragma unroll
            for (int kk = 0; kk < 4; kk++)
#pragma unroll
                for (int q = 0; q < RM / 4; q++) { const float4 v = *reinterpret_cast<const float4 *>(As + (k + kk) * PA_R + q * 16 + lr * 4); a[4 * q][kk] = v.x; a[4 * q + 1][kk] = v.y; a[4 * q + 2][kk] = v.z; a[4 * q + 3][kk] = v.w; }
        }
        if (b_kc) {
#pragma unroll
            for (int c = 0; c < RN; c++) { const float4 v = *reinterpret_cast<const float4 *>(Bs + (lc + 8 * c) * PB_K + k); b[c][0] = v.x; b[c][1] = v.y; b[c][2] = v.z; b[c][3] = v.w; }
        } else {
#pragma unroll
            for (int kk = 0; kk < 4; kk++)
#pragma unroll
                for (int q = 0; q < RN / 4; q++) { const float4 v = *reinterpret_cast<const float4 *>(Bs + (k + kk) * PB_R + q * 32 + lc * 4); b[4 * q][kk] = v.x; b[4 * q + 1][kk] = v.y; b[4 * q + 2][kk] = v.z; b[4 * q + 3][kk] = v.w; }
        }
#pragma unroll
        for (int kk = 0; kk < 4; kk++)
#pragma unroll
            for (int r = 0; r < RM; r++)
#pragma unroll
                for (int c = 0; c < RN; c++) acc[r][c] = fmaf(a[r][kk], b[c][kk], acc[r][c]);
    }
}

__device__ __forceinline__ void gg_ldsm(uint32_t (&r)[4], uint32_t addr) { asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr)); }
__device__ __forceinline__ void gg_ldsm_t(uint32_t (&r)[4], uint32_t addr) { asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr)); }
__device__ __forceinline__ void gg_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// fp16: one k16 step of a warp tile of MI x 16 rows and NI x 16 columns
template <bool a_kc, bool b_kc, int MI, int NI, int PA_K, int PA_R, int PB_K, int PB_R>
__device__ __forceinline__ void gg_hmma(uint32_t As, uint32_t Bs, int row0, int col0, int k0, float (&acc)[MI][2 * NI][4], int lane)
{
    uint32_t a[MI][4], b[NI][4];
    const int l8 = lane & 7, h1 = (lane >> 3) & 1, h2 = lane >> 4;
    if (a_kc) {
#pragma unroll
        for (int i = 0; i < MI; i++) gg_ldsm(a[i], As + (uint32_t)((row0 + 16 * i + l8 + 8 * h1) * PA_K + k0 + 8 * h2) * 2u);
    } else {
#pragma unroll
        for (int i = 0; i < MI; i++) gg_ldsm_t(a[i], As + (uint32_t)((k0 + l8 + 8 * h2) * PA_R + row0 + 16 * i + 8 * h1) * 2u);
    }
    if (b_kc) {
#pragma unroll
        for (int j = 0; j < NI; j++) gg_ldsm(b[j], Bs + (uint32_t)((col0 + 16 * j + l8 + 8 * h2) * PB_K + k0 + 8 * h1) * 2u);
    } else {
#pragma unroll
        for (int j = 0; j < NI; j++) gg_ldsm_t(b[j], Bs + (uint32_t)((k0 + l8 + 8 * h1) * PB_R + col0 + 16 * j + 8 * h2) * 2u);
    }
#pragma unroll
    for (int i = 0; i < MI; i++)
#pragma unroll
        for (int j = 0; j < NI; j++) { gg_mma(acc[i][2 * j], a[i], b[j][0], b[j][1]); gg_mma(acc[i][2 * j + 1], a[i], b[j][2], b[j][3]); }
}

// BM x BN tile of C; WM x WN warps side by side over the tile, WK warps over the K steps of a chunk of KC.
template <class T, int BM, int BN, int WM, int WN, int WK, int KC, int ST> struct GgCfg {
    static constexpr int NT = 32 * WM * WN * WK;
    static constexpr int PAD = 16 / (int)sizeof(T);                        // 16-byte rows that do not repeat in the banks
    static constexpr int PK = KC + PAD, PA_R = BM + PAD, PB_R = BN + PAD;
    static constexpr int A_EL = BM * PK > KC * PA_R ? BM * PK : KC * PA_R, B_EL = BN * PK > KC * PB_R ? BN * PK : KC * PB_R;
    static constexpr int STAGE = A_EL + B_EL;                              // elements
    static constexpr int RED_P = BN + 4;                                   // floats per row of a partial tile
    static constexpr size_t SMEM_OP = (size_t)ST * STAGE * sizeof(T), SMEM_RED = (size_t)WK * BM * RED_P * 4;
    static constexpr size_t SMEM = SMEM_OP > SMEM_RED ? SMEM_OP : SMEM_RED;
};

template <class T, int BM, int BN, int WM, int WN, int WK, int KC, int ST, int OCC, int G>
__global__ void __launch_bounds__(32 * WM * WN * WK, OCC) gemm_group_kernel(const __grid_constant__ GgParams<T, G> g)
{
    typedef GgCfg<T, BM, BN, WM, WN, WK, KC, ST> Cfg;
    constexpr int NT = Cfg::NT, PAD = Cfg::PAD, PK = Cfg::PK, PA_R = Cfg::PA_R, PB_R = Cfg::PB_R;
    extern __shared__ __align__(16) unsigned char gg_smem[];
    T *ops = reinterpret_cast<T *>(gg_smem);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

    int pi = 0;
#pragma unroll
    for (int i = 1; i < G; i++) pi += (int)blockIdx.x >= g.first[i];
    const GgProb<T> &p = g.p[G == 1 ? 0 : pi];
    const int local = (int)blockIdx.x - (G == 1 ? 0 : g.first[pi]);
    const int tile = gg_quot(local, p.splits), split = local - tile * p.splits.d;
    const int b = gg_quot(tile, p.tiles_nm), t2 = tile - b * p.tiles_nm.d, trow = gg_quot(t2, p.tiles_m);
    const int i0 = trow * BM, j0 = (t2 - trow * p.tiles_m.d) * BN;
    const int a_kc = p.a_kc, b_kc = p.b_kc;
    const int ch0 = split * p.per, nch = min(p.chunks - ch0, p.per);
    const int K = p.K, cps = p.cps.d;                                      // chunks of a segment

    // walk of the copies: chunk within its segment, segment
    GgLoader<T, BM, KC, PAD, NT> la;
    GgLoader<T, BN, KC, PAD, NT> lb;
    int f_seg = gg_quot(ch0, p.cps), f_c = ch0 - f_seg * cps, f_left = nch;
    const int c_first = f_c;
    auto open_segment = [&]() {
        const T *A, *B;
        if (p.seg_list) { A = f_seg == 0 ? p.A[0] : f_seg == 1 ? p.A[1] : p.A[2]; B = f_seg == 0 ? p.B[0] : f_seg == 1 ? p.B[1] : p.B[2]; }
        else { A = p.A[0] + f_seg * p.a_ks; B = p.B[0] + f_seg * p.b_ks; }
        la.init(A + b * p.a_bs, a_kc, p.a_vl, i0, f_c * KC, p.N, p.a_cs, p.a_ss_);
        lb.init(B + b * p.b_bs, b_kc, p.b_vl, j0, f_c * KC, p.M, p.b_cs, p.b_ss_);
    };
    open_segment();
    // what the end of the kernel reads of its parameters: a first read of one misses the constant cache
    asm volatile("" ::"l"(p.C), "l"(p.c_bs), "l"(p.c_rs), "l"(p.c_cs), "f"(p.alpha), "r"(p.plain));
    const int nsplits = p.splits.d;
    pdl_wait();                                                            // everything above reads parameters only
    const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(gg_smem);
    auto fetch = [&](int stage) {
        if (f_left > 0) {
            const uint32_t st = sbase + (uint32_t)(stage * Cfg::STAGE * (int)sizeof(T));
            la.fetch(st, K - f_c * KC);
            lb.fetch(st + (uint32_t)(Cfg::A_EL * (int)sizeof(T)), K - f_c * KC);
            f_left--;
            if (++f_c == cps && f_left > 0) { f_c = 0; f_seg++; open_segment(); }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    const int wk = warp / (WM * WN), wmn = warp % (WM * WN), wm = wmn / WN, wn = wmn % WN;
    constexpr int TM = BM / WM, TN = BN / WN;                              // warp tile
    constexpr int RM = TM / 4, RN = TN / 8, MI = TM / 16, NI = TN / 16;
    constexpr bool HALF = sizeof(T) == 2;
    float accf[HALF ? 1 : RM][HALF ? 1 : RN];
    float acch[HALF ? MI : 1][HALF ? 2 * NI : 1][4];
    if constexpr (HALF) {
#pragma unroll
        for (int i = 0; i < MI; i++)
#pragma unroll
            for (int j = 0; j < 2 * NI; j++)
#pragma unroll
                for (int q = 0; q < 4; q++) acch[i][j][q] = 0.f;
    } else {
#pragma unroll
        for (int r = 0; r < RM; r++)
#pragma unroll
            for (int c = 0; c < RN; c++) accf[r][c] = 0.f;
    }

    for (int s = 0; s < ST - 1; s++) fetch(s);
    int cur = 0, c_c = c_first;
    for (int ch = 0; ch < nch; ch++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(ST - 2) : "memory");
        __syncthreads();
        fetch(cur == 0 ? ST - 1 : cur - 1);
        const T *as = ops + cur * Cfg::STAGE, *bs = as + Cfg::A_EL;
        // K steps past the end of the segment hold zeros: skip them
        const int k_live = K - c_c * KC;
        if (++c_c == cps) c_c = 0;
        // one copy of the arithmetic per pair of layouts: the operand registers are never merged across branches
        auto multiply = [&](auto akc, auto bkc) {
            constexpr bool AK = decltype(akc)::value, BK = decltype(bkc)::value;
            if constexpr (HALF) {
                const uint32_t au = (uint32_t)__cvta_generic_to_shared(as), bu = (uint32_t)__cvta_generic_to_shared(bs);
#pragma unroll
                for (int k = 16 * wk; k < KC; k += 16 * WK)
                    if (k < k_live) gg_hmma<AK, BK, MI, NI, PK, PA_R, PK, PB_R>(au, bu, wm * TM, wn * TN, k, acch, lane);
            } else {
                constexpr int KW = KC / WK;
                if (wk * KW < k_live)
                    gg_ffma<AK, BK, RM, RN, PK, PA_R, PK, PB_R, KW>(as + wm * TM * (AK ? PK : 1), bs + wn * TN * (BK ? PK : 1), wk * KW, accf, lane >> 3, lane & 7);
            }
        };
        if (a_kc) { if (b_kc) multiply(std::true_type(), std::true_type()); else multiply(std::true_type(), std::false_type()); }
        else { if (b_kc) multiply(std::false_type(), std::true_type()); else multiply(std::false_type(), std::false_type()); }
        cur = cur + 1 == ST ? 0 : cur + 1;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();

    // partial tiles of the K warps meet in shared memory
    float *red = reinterpret_cast<float *>(gg_smem);
    float *mine = red + wk * BM * Cfg::RED_P;
    if constexpr (HALF) {
#pragma unroll
        for (int i = 0; i < MI; i++)
#pragma unroll
            for (int j = 0; j < 2 * NI; j++) {
                const int r = wm * TM + 16 * i + (lane >> 2), c = wn * TN + 8 * j + 2 * (lane & 3);
                *reinterpret_cast<float2 *>(mine + r * Cfg::RED_P + c) = make_float2(acch[i][j][0], acch[i][j][1]);
                *reinterpret_cast<float2 *>(mine + (r + 8) * Cfg::RED_P + c) = make_float2(acch[i][j][2], acch[i][j][3]);
            }
    } else {
        const int lr = lane >> 3, lc = lane & 7;
#pragma unroll
        for (int r = 0; r < RM; r++)
#pragma unroll
            for (int c = 0; c < RN; c++) mine[(wm * TM + gg_row<RM>(r, lr, a_kc)) * Cfg::RED_P + wn * TN + gg_col<RN>(c, lc, b_kc)] = accf[r][c];
    }
    __syncthreads();

    constexpr int Q = BN / 4, QUADS = BM * Q;                              // four neighbouring columns per thread
    if (nsplits > 1) {
        __shared__ unsigned ticket_s;
        float *part = p.part + ((size_t)tile * nsplits + split) * (BM * BN);
        for (int e = tid; e < QUADS; e += NT) {
            const int i = e / Q, j = (e % Q) * 4;
            float4 v = *reinterpret_cast<const float4 *>(red + i * Cfg::RED_P + j);
#pragma unroll
            for (int w = 1; w < WK; w++) { const float4 u = *reinterpret_cast<const float4 *>(red + (w * BM + i) * Cfg::RED_P + j); v.x += u.x; v.y += u.y; v.z += u.z; v.w += u.w; }
            __stcg(reinterpret_cast<float4 *>(part) + e, v);
        }
        __threadfence();
        __syncthreads();
        if (tid == 0) ticket_s = atomicAdd(&gg_tickets[p.ticket0 + tile], 1u);
        __syncthreads();
        if (ticket_s != (unsigned)(nsplits - 1)) return;
        __threadfence();
        if (tid == 0) gg_tickets[p.ticket0 + tile] = 0;
    }
    T *C = p.C + b * p.c_bs;
    const long long c_rs = p.c_rs, c_cs = p.c_cs;
    const float alpha = p.alpha;
    const int plain = p.plain;
    for (int e = tid; e < QUADS; e += NT) {
        const int i = e / Q, j = (e % Q) * 4;
        if (i0 + i >= p.N || j0 + j >= p.M) continue;
        float4 v;
        if (nsplits > 1) {
            const float4 *src = reinterpret_cast<const float4 *>(p.part + (size_t)tile * nsplits * (BM * BN)) + e;
            v = __ldcg(src);
#pragma unroll 4
            for (int s = 1; s < nsplits; s++) { const float4 u = __ldcg(src + (size_t)s * QUADS); v.x += u.x; v.y += u.y; v.z += u.z; v.w += u.w; }
        } else {
            v = *reinterpret_cast<const float4 *>(red + i * Cfg::RED_P + j);
#pragma unroll
            for (int w = 1; w < WK; w++) { const float4 u = *reinterpret_cast<const float4 *>(red + (w * BM + i) * Cfg::RED_P + j); v.x += u.x; v.y += u.y; v.z += u.z; v.w += u.w; }
        }
        float r[4] = {v.x * alpha, v.y * alpha, v.z * alpha, v.w * alpha};
        T *dst = C + (long long)(i0 + i) * c_rs + (long long)(j0 + j) * c_cs;
        const int live = min(4, p.M - j0 - j);
        bool whole = plain && live == 4;
        if (!whole) {
            const float brow = p.bias_mode == 1 ? ld(p.bias + i0 + i) : 0.f;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                if (q >= live) break;
                if (p.accumulate) r[q] += ld(dst + q * c_cs);
                if (p.bias_mode == 1) r[q] += brow; else if (p.bias_mode == 2) r[q] += ld(p.bias + j0 + j + q);
            }
            whole = p.quads && live == 4;
            if (!whole) {
#pragma unroll
                for (int q = 0; q < 4; q++) if (q < live) st(dst + q * c_cs, r[q]);
            }
        }
        if (!whole) continue;
        if constexpr (HALF) {
            __half2 h0 = __floats2half2_rn(r[0], r[1]), h1 = __floats2half2_rn(r[2], r[3]);
            *reinterpret_cast<uint2 *>(dst) = make_uint2(*reinterpret_cast<uint32_t *>(&h0), *reinterpret_cast<uint32_t *>(&h1));
        } else *reinterpret_cast<float4 *>(dst) = make_float4(r[0], r[1], r[2], r[3]);
    }
}

// ---------------------------------------------------------------- host side
// Which of an operand's two indices runs along shared-memory rows, and how wide its copies may be.
template <class T> static void gg_operand(const T *const *ptrs, int nptr, long long rs, long long ks, long long bs, int batch, long long seg, int segs, bool list,
                                          int &kc, int &vl, long long &cs, long long &ss)
{
    kc = ks == 1 || (rs != 1 && std::llabs(ks) <= std::llabs(rs));
    cs = kc ? ks : rs; ss = kc ? rs : ks;
    constexpr int V16 = 16 / (int)sizeof(T), V4 = 4 / (int)sizeof(T);
    vl = 0;                                                                // one element
    if (cs != 1) return;
    auto fits = [&](int v) {
        const size_t mask = (size_t)v * sizeof(T) - 1;
        for (int i = 0; i < nptr; i++) if (((uintptr_t)ptrs[i]) & mask) return false;
        return ss % v == 0 && (batch == 1 || bs % v == 0) && (list || segs == 1 || seg % v == 0);
    };
    if (fits(V16)) vl = sizeof(T) == 4 ? 2 : 3; else if (V4 > 1 && fits(V4)) vl = 1;
}

// What a chunk of an operand costs beyond that of 16-byte copies: more of them, and single halves come by way of registers, eight loads in
// flight at a time (175 x 869 x 60 with rows of 869 halves: 10.1 us with no split, 5.8 with the ones that this asks for).
template <class T, int ROWS, int KC, int NT> static constexpr int gg_copy_cycles(int vl)
{
    constexpr int V16 = 16 / (int)sizeof(T), V4 = 4 / (int)sizeof(T);
    return (1 << vl) == V16 ? 0 : (1 << vl) == V4 ? ROWS * KC / V4 / NT * 8 : ROWS * KC / NT / 8 * 200;
}

// CYC: cycles of one K chunk in a CTA (measured with the SMs about as full as such products make them), in units of those of a split:
// writing the partial tile, the ticket and the last CTA's sum cost 2500 cycles, and 150 more per split.
template <class T, int BM, int BN, int WM, int WN, int WK, int KC, int ST, int OCC, int CYC, int G>
static void gg_launch(Scope &sc, const GemmGroup<T> *list, int count)
{
    typedef GgCfg<T, BM, BN, WM, WN, WK, KC, ST> Cfg;
    GgParams<T, G> g;
    for (int i = 0; i < G; i++) g.first[i] = 0x7fffffff;
    int tiles_of[GG_MAX];
    long long tiles_all = 0, tile_steps = 0;
    int shortest = 1 << 30;
    for (int i = 0; i < count; i++) {
        const GemmGroup<T> &s = list[i];
        GgProb<T> &p = g.p[i];
        const bool tr = s.c_cs != 1 && s.c_rs == 1;                        // column-major result: compute its transpose
        for (int q = 0; q < 3; q++) { p.A[q] = tr ? s.B[q] : s.A[q]; p.B[q] = tr ? s.A[q] : s.B[q]; }
        p.C = s.C; p.bias = s.bias;
        p.N = tr ? s.M : s.N; p.M = tr ? s.N : s.M; p.K = s.K; p.segs = s.segs; p.seg_list = s.seg_list;
        const long long a_rs = tr ? s.b_cs : s.a_rs, a_ks_ = tr ? s.b_rs : s.a_cs, b_rs_ = tr ? s.a_rs : s.b_cs, b_ks_ = tr ? s.a_cs : s.b_rs;
        p.a_bs = tr ? s.b_bs : s.a_bs; p.b_bs = tr ? s.a_bs : s.b_bs; p.c_bs = s.c_bs;
        p.a_ks = tr ? s.b_ks : s.a_ks; p.b_ks = tr ? s.a_ks : s.b_ks;
        p.c_rs = tr ? s.c_cs : s.c_rs; p.c_cs = tr ? s.c_rs : s.c_cs;
        const int np = s.seg_list ? s.segs : 1;
        gg_operand<T>(p.A, np, a_rs, a_ks_, p.a_bs, s.batch, p.a_ks, s.segs, s.seg_list != 0, p.a_kc, p.a_vl, p.a_cs, p.a_ss_);
        gg_operand<T>(p.B, np, b_rs_, b_ks_, p.b_bs, s.batch, p.b_ks, s.segs, s.seg_list != 0, p.b_kc, p.b_vl, p.b_cs, p.b_ss_);
        p.alpha = s.alpha; p.accumulate = s.accumulate ? 1 : 0;
        p.bias_mode = s.bias ? (tr && s.bias_mode ? 3 - s.bias_mode : s.bias_mode) : 0;
        const int tiles_m = ceil_div(p.M, BN);
        tiles_of[i] = tiles_m * ceil_div(p.N, BM);
        p.tiles_m = gg_div(std::max(1, tiles_m), tiles_of[i]); p.tiles_nm = gg_div(tiles_of[i], (long long)tiles_of[i] * s.batch);
        p.chunks = p.segs * ceil_div(p.K, KC); p.cps = gg_div(std::max(1, ceil_div(p.K, KC)), p.chunks);
        p.quads = p.c_cs == 1 && (p.c_rs & 3) == 0 && (s.batch == 1 || (p.c_bs & 3) == 0) && (((uintptr_t)p.C) & (4 * sizeof(T) - 1)) == 0;
        p.plain = p.quads && !p.accumulate && !p.bias_mode;
        p.part = nullptr; p.ticket0 = 0;
        tiles_all += (long long)tiles_of[i] * s.batch;
        shortest = std::min(shortest, p.chunks);
        tile_steps += (long long)tiles_of[i] * s.batch * p.chunks;
    }
    // Split K over CTAs while the group leaves SMs idle, up to enough CTAs for two per SM, and only as far as the chunks saved are worth it
    // (128 x 512 x 128 in fp16, 32 tiles: two splits 6300 cycles, none 4700).
    const long long want = 2ll * sm_count();
    int ticket = 0;
    long long first = 0;
    for (int i = 0; i < count; i++) {
        GgProb<T> &p = g.p[i];
        const long long tiles = (long long)tiles_of[i] * list[i].batch;
        int splits = 1;
        // this product's share of the wanted CTAs, per tile; in a group that fills the SMs, a contraction much longer than the
        // shortest one (three segments beside products of one) is cut to about that length
        const bool filled = tiles_all >= sm_count();
        const long long most = !filled ? (want * p.chunks + tile_steps - 1) / std::max(1ll, tile_steps) : (tiles_all < 4 * sm_count() && p.chunks >= 2 * shortest ? p.chunks / std::max(shortest, 1) : 1);
        if (most > 1 && p.chunks >= 2) {
            const int cap = (int)std::min<long long>(std::min<long long>(most, p.chunks), 64);
            const long long cyc = CYC + gg_copy_cycles<T, BM, KC, Cfg::NT>(p.a_vl) + gg_copy_cycles<T, BN, KC, Cfg::NT>(p.b_vl);
            long long best = p.chunks * cyc;
            for (int s = 2; s <= cap; s++) {
                const int per = ceil_div(p.chunks, s);
                const long long cost = per * cyc + 2500 + 150 * s;
                if (cost < best) { best = cost; splits = ceil_div(p.chunks, per); }
            }
            if (splits > 1) {
                if (ticket + tiles <= 16384) p.part = sc.try_scratch<float>((size_t)tiles * splits * BM * BN);
                if (p.part) { p.ticket0 = ticket; ticket += (int)tiles; }
                else splits = 1;
            }
        }
        p.splits = gg_div(splits, tiles * splits); p.per = ceil_div(p.chunks, splits);
        g.first[i] = (int)first;
        first += tiles * splits;
    }
    auto kern = gemm_group_kernel<T, BM, BN, WM, WN, WK, KC, ST, OCC, G>;
    static bool attr_set = false;
    if (!attr_set) { cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Cfg::SMEM); attr_set = true; }
    TL_LAUNCH((gemm_group_kernel<T, BM, BN, WM, WN, WK, KC, ST, OCC, G>), (unsigned)first, Cfg::NT, Cfg::SMEM, g);
}

template <class T> void gemm_group(const GemmGroup<T> *list, int count)
{
    GemmGroup<T> live[GG_MAX];
    int n = 0;
    if (count > GG_MAX) { set_error(TL_ERR_BAD_ARGS, "gemm_group: %d products (%d at most)", count, GG_MAX); return; }
    long long tiles64 = 0, tiles32 = 0;
    for (int i = 0; i < count; i++) {
        if (list[i].N <= 0 || list[i].M <= 0 || list[i].batch <= 0) continue;
        live[n++] = list[i];
        tiles64 += (long long)ceil_div(list[i].N, 64) * ceil_div(list[i].M, 64) * list[i].batch;
        tiles32 += (long long)ceil_div(list[i].N, 32) * ceil_div(list[i].M, 32) * list[i].batch;
    }
    if (!n) return;
    Scope sc;
    if (!sc.ok()) return;
    // Tiles by how many of them the group has (measured over 256^3, 300x400x500, 16x2048x4096, 17x3000x40, 2000x64x300 ...):
    // small tiles while they are needed to occupy the SMs, larger ones as soon as they come to about one and a half per SM.
    // fp32, us: 256^3 4.8 with 16 x 32 tiles, 6.1 with 32 x 32; 2000x50x2000 46 and 35.  fp16: 128x512x128 4.9 with 16 x 32,
    // 5.7 with 32 x 32, 9.7 with 64 x 64; 1000x60x1000 11.8, 10.3, 6.4.  Four warps per CTA, several CTAs per SM: eight warps
    // on one 32 x 32 fp32 tile cost 20 to 40 % more (shorter runs of FMAs between barriers).
#define GG_LAUNCH(...) do { if (n == 1) gg_launch<T, __VA_ARGS__, 1>(sc, live, n); else gg_launch<T, __VA_ARGS__, GG_MAX>(sc, live, n); } while (0)
    if constexpr (sizeof(T) == 2) {
        if (tiles64 >= sm_count()) GG_LAUNCH(64, 64, 2, 2, 1, 64, 3, 3, 900);
        else if (tiles32 >= sm_count()) GG_LAUNCH(32, 32, 1, 1, 4, 128, 3, 4, 700);
        else GG_LAUNCH(16, 32, 1, 1, 4, 128, 3, 4, 500);
    } else {
        if (2 * tiles32 >= 3 * sm_count()) GG_LAUNCH(32, 32, 2, 1, 2, 64, 3, 4, 2500);
        else GG_LAUNCH(16, 32, 1, 1, 4, 64, 3, 4, 1200);
    }
#undef GG_LAUNCH
}
template void gemm_group<float>(const GemmGroup<float> *, int);
template void gemm_group<__half>(const GemmGroup<__half> *, int);

} // namespace tl

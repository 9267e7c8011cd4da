// Fused attention core of the multi-head self-attention layer.
//
// Forward: one kernel per (head, tile of queries) forms the scaled scores q^T k of its queries against all keys in
// shared memory, takes the row softmax there, writes the probabilities P once (the reference keeps them for the
// backward pass, so they are an output of the layer) and multiplies them with v before leaving: the scores never
// reach HBM and P is not read back  [ref: lib/sources/pulp_mhsa_fp32.c:348-560: per head a transpose, a matmul, a
// scalar multiply, a transpose, a softmax, a transpose and a matmul, each through memory].
//
// Backward: two kernels.  The query-tiled one recomputes nothing it can keep: dP = datt^T v for its queries is formed
// in shared memory (and written, because the reference exposes it as softmax_buffer.diff), turned into
// dS = (dP - sum_key dP P) P in place, and contracted with k into dq; it also leaves the row sums sum_key dP P behind.
// The key-tiled one rebuilds its columns of dS from P, dP and those row sums and contracts them with q and datt into
// dk and dv.  dS never reaches HBM  [ref: lib/sources/pulp_mhsa_fp32.c:842-1400].
//
// Layouts (reference convention): q, k, v, att and their gradients are F x L (token index fastest, head h owns rows
// h*H .. h*H+H-1); P and dP are heads x L x L indexed [head][query][key].  Every sum runs in a fixed order.
#include "tl_kernels.h"
#include "tl_reduce.cuh"
#include "tl_tc.cuh"

namespace tl {

// What bounds these kernels is latency: the arithmetic of four heads x 256 tokens x 64 is a microsecond of the chip's FMAs, the
// operands come from L2.  So every loop fetches a batch of independent elements before it uses the first (16 rows of k per
// thread, four rows of v times four column blocks per lane), and a warp takes four rows at once so that what it reads of the
// tile in shared memory serves all of them and their sixteen sums fold in one butterfly.  Measured, fp32, 4 heads x 256 x 64:
// forward 15.0 -> 9.8 us, query half 11.6 -> 9.5, key half 15.3 -> 8.7.
static constexpr int ATT_THREADS = 256;
static constexpr int ATT_TQ = 4;                 // queries (or keys) per CTA = accumulators per thread.  Four: 256 CTAs for 4 heads x 256
                                                 // tokens, two per SM on most SMs; with eight (128 CTAs of 8 warps) the kernels ran at an eighth of the warp slots
static constexpr int ATT_ROWS = 4;               // rows of M per warp and pass in rows_times_tile

// tile[t][j] = alpha * sum_d a_tile[d][t] * M[d][j]  for t < ATT_TQ, j < L: thread per column j, the H-long contraction in
// registers.  a_tile is [H][ATT_TQ] in shared memory (broadcast reads), M rows are read coalesced.
template <class T>
__device__ __forceinline__ void tile_from_rows(const float *a_tile, const T *__restrict__ M, float *tile, int Lp, int H, int L, float alpha)
{
    constexpr int B = 16;
    for (int j = threadIdx.x; j < L; j += ATT_THREADS) {
        float acc[ATT_TQ] = {0.f, 0.f, 0.f, 0.f};
        for (int d0 = 0; d0 < H; d0 += B) {
            float m[B];
            if constexpr (sizeof(T) == 4) {
#pragma unroll
                for (int u = 0; u < B; u++) m[u] = d0 + u < H ? M[(size_t)(d0 + u) * L + j] : 0.f;
            } else {
                // rows past the last are fetched from it and replaced by zero: under a condition, a load and its conversion from half
                // precision were waited for one by one (16 x 240 cycles); in fp32 the clamps cost more than they save
                T raw[B];
#pragma unroll
                for (int u = 0; u < B; u++) raw[u] = M[(size_t)min(d0 + u, H - 1) * L + j];
#pragma unroll
                for (int u = 0; u < B; u++) m[u] = d0 + u < H ? __half2float(raw[u]) : 0.f;
            }
#pragma unroll
            for (int u = 0; u < B; u++) {
                const float4 a = *reinterpret_cast<const float4 *>(a_tile + min(d0 + u, H - 1) * ATT_TQ);
                acc[0] = fmaf(a.x, m[u], acc[0]); acc[1] = fmaf(a.y, m[u], acc[1]); acc[2] = fmaf(a.z, m[u], acc[2]); acc[3] = fmaf(a.w, m[u], acc[3]);
            }
        }
#pragma unroll
        for (int t = 0; t < ATT_TQ; t++) tile[t * Lp + j] = __fmul_rn(acc[t], alpha);
    }
}

// out[d][t0 + t] = alpha * sum_j M[d][j] * tile[t][j]  for d < H, t < nt: a warp per four rows d, lanes over j (coalesced reads
// of M, conflict-free reads of the tile); lanes 2 (4 r + t) and 2 (4 r + t) + 1 end up with the sum of row r and column t.
template <class T>
__device__ __forceinline__ void rows_times_tile(const T *__restrict__ M, const float *tile, int Lp, int H, int L, T *__restrict__ out, int t0, int nt, float alpha)
{
    constexpr int R = ATT_ROWS, U = 4;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int d0 = warp * R; d0 < H; d0 += (ATT_THREADS / 32) * R) {
        const T *row[R];
#pragma unroll
        for (int r = 0; r < R; r++) row[r] = M + (size_t)min(d0 + r, H - 1) * L;
        float acc[R * ATT_TQ];
#pragma unroll
        for (int i = 0; i < R * ATT_TQ; i++) acc[i] = 0.f;
        for (int j0 = 0; j0 < L; j0 += 32 * U) {
            float m[U][R];
            if constexpr (sizeof(T) == 4) {
#pragma unroll
                for (int u = 0; u < U; u++)
#pragma unroll
                    for (int r = 0; r < R; r++) m[u][r] = j0 + 32 * u + lane < L ? row[r][j0 + 32 * u + lane] : 0.f;
            } else {
                T raw[U][R];
#pragma unroll
                for (int u = 0; u < U; u++)
#pragma unroll
                    for (int r = 0; r < R; r++) raw[u][r] = row[r][min(j0 + 32 * u + lane, L - 1)];
#pragma unroll
                for (int u = 0; u < U; u++)
#pragma unroll
                    for (int r = 0; r < R; r++) m[u][r] = j0 + 32 * u + lane < L ? __half2float(raw[u][r]) : 0.f;
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                if (j0 + 32 * u >= L) break;
                const int j = min(j0 + 32 * u + lane, L - 1);
#pragma unroll
                for (int t = 0; t < ATT_TQ; t++) {
                    const float c = tile[t * Lp + j];
#pragma unroll
                    for (int r = 0; r < R; r++) acc[r * ATT_TQ + t] = fmaf(m[u][r], c, acc[r * ATT_TQ + t]);
                }
            }
        }
        // fold: after the step of offset o a lane keeps the half of its sums that its bit of o selects
#pragma unroll
        for (int o = 16, n = 8; o > 1; o >>= 1, n >>= 1)
#pragma unroll
            for (int i = 0; i < 8; i++)
                if (i < n) {
                    const float keep = (lane & o) ? acc[i + n] : acc[i], send = (lane & o) ? acc[i] : acc[i + n];
                    acc[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                }
        const float sum = acc[0] + __shfl_xor_sync(0xffffffffu, acc[0], 1);
        const int r = lane >> 3, t = (lane >> 1) & 3;
        if ((lane & 1) == 0 && d0 + r < H && t < nt) st(out + (size_t)(d0 + r) * L + t0 + t, __fmul_rn(sum, alpha));
    }
}

// four neighbours from a 4-element-aligned address
__device__ __forceinline__ void ld4(const float *p, float (&v)[4]) { const float4 x = *reinterpret_cast<const float4 *>(p); v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w; }
__device__ __forceinline__ void ld4(const __half *p, float (&v)[4])
{
    const uint2 x = *reinterpret_cast<const uint2 *>(p);
    const float2 a = __half22float2(*reinterpret_cast<const __half2 *>(&x.x)), b = __half22float2(*reinterpret_cast<const __half2 *>(&x.y));
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
// a_tile[d][t] = A[d][t0 + t] (zero beyond the last token)
template <class T>
__device__ __forceinline__ void load_a_tile(const T *__restrict__ A, float *a_tile, int H, int L, int t0)
{
    for (int i = threadIdx.x; i < H * ATT_TQ; i += ATT_THREADS) {
        const int d = i / ATT_TQ, t = i % ATT_TQ;
        a_tile[i] = ld0(t0 + t < L, A + (size_t)d * L + t0 + t);
    }
}

template <class T>
__global__ void __launch_bounds__(ATT_THREADS) attn_fw_kernel(const T *__restrict__ q, const T *__restrict__ k, const T *__restrict__ v,
                                                              T *__restrict__ P, T *__restrict__ att, int L, int H, float scaling)
{
    pdl_wait();
    extern __shared__ __align__(16) float att_smem[];
    const int Lp = L + 1, head = blockIdx.y, t0 = blockIdx.x * ATT_TQ, nt = min(ATT_TQ, L - t0);
    float *a_tile = att_smem, *tile = att_smem + H * ATT_TQ;
    const size_t hoff = (size_t)head * H * L;
    load_a_tile(q + hoff, a_tile, H, L, t0);
    __syncthreads();
    tile_from_rows(a_tile, k + hoff, tile, Lp, H, L, scaling);
    __syncthreads();
    // row softmax, a warp per query: max, Schraudolph exp of (x - max), divide by the row sum  [ref: pulp_act_fp32.c:187-245]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp < nt) {
        float *row = tile + warp * Lp;
        float m = -FLT_MAX;
        for (int j = lane; j < L; j += 32) m = fmaxf(m, row[j]);
        m = warp_max(m);
        float s = 0.f;
        for (int j = lane; j < L; j += 32) { const float e = fastexp_gist_dev(__fsub_rn(row[j], m)); row[j] = e; s += e; }
        s = warp_sum(s);
        T *prow = P + ((size_t)head * L + t0 + warp) * L;
        for (int j = lane; j < L; j += 32) { const float p = __fdiv_rn(row[j], s); row[j] = p; st(prow + j, p); }
    } else if (warp < ATT_TQ) {
        float *row = tile + warp * Lp;
        for (int j = lane; j < L; j += 32) row[j] = 0.f;
    }
    __syncthreads();
    rows_times_tile(v + hoff, tile, Lp, H, L, att + hoff, t0, nt, 1.0f);
}

// Query-tiled half of the backward pass: dP (written), row sums of dP * P (written), dq (written).
template <class T>
__global__ void __launch_bounds__(ATT_THREADS) attn_bw_query_kernel(const T *__restrict__ datt, const T *__restrict__ v, const T *__restrict__ k,
                                                                    const T *__restrict__ P, T *__restrict__ dP, float *__restrict__ rowdot,
                                                                    T *__restrict__ dq, int L, int H, float scaling)
{
    pdl_wait();
    extern __shared__ __align__(16) float att_smem[];
    const int Lp = L + 1, head = blockIdx.y, t0 = blockIdx.x * ATT_TQ, nt = min(ATT_TQ, L - t0);
    float *a_tile = att_smem, *tile = att_smem + H * ATT_TQ;
    const size_t hoff = (size_t)head * H * L;
    load_a_tile(datt + hoff, a_tile, H, L, t0);
    __syncthreads();
    tile_from_rows(a_tile, v + hoff, tile, Lp, H, L, 1.0f);
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp < nt) {
        // dS = (dP - sum_key dP P) P   [ref: lib/sources/pulp_act_fp32.c:335-392]
        float *row = tile + warp * Lp;
        const size_t roff = ((size_t)head * L + t0 + warp) * L;
        float s = 0.f;
        for (int j0 = 0; j0 < L; j0 += 256) {
            float p[8];
#pragma unroll
            for (int u = 0; u < 8; u++) p[u] = ld0(j0 + 32 * u + lane < L, P + roff + j0 + 32 * u + lane);
#pragma unroll
            for (int u = 0; u < 8; u++) {
                const int j = j0 + 32 * u + lane;
                if (j >= L) break;
                float g = row[j];
                if (sizeof(T) == 2) g = __half2float(__float2half_rn(g));          // the value the caller sees in dP
                st(dP + roff + j, g);
                s = fmaf(g, p[u], s);
            }
        }
        s = warp_sum(s);
        if (lane == 0) rowdot[(size_t)head * L + t0 + warp] = s;
        for (int j0 = 0; j0 < L; j0 += 256) {
            float p[8];
#pragma unroll
            for (int u = 0; u < 8; u++) p[u] = ld0(j0 + 32 * u + lane < L, P + roff + j0 + 32 * u + lane);
#pragma unroll
            for (int u = 0; u < 8; u++) {
                const int j = j0 + 32 * u + lane;
                if (j >= L) break;
                float g = row[j];
                if (sizeof(T) == 2) g = __half2float(__float2half_rn(g));
                row[j] = __fmul_rn(__fsub_rn(g, s), p[u]);
            }
        }
    } else if (warp < ATT_TQ) {
        float *row = tile + warp * Lp;
        for (int j = lane; j < L; j += 32) row[j] = 0.f;
    }
    __syncthreads();
    rows_times_tile(k + hoff, tile, Lp, H, L, dq + hoff, t0, nt, scaling);
}

// Key-tiled half: columns of P and of dS = (dP - rowdot) P for ATT_TQ keys against all queries, then
// dv[d][key] = sum_query datt[d][query] P[query][key] and dk[d][key] = scaling * sum_query q[d][query] dS[query][key].
template <class T>
__global__ void __launch_bounds__(ATT_THREADS) attn_bw_key_kernel(const T *__restrict__ datt, const T *__restrict__ q, const T *__restrict__ P,
                                                                  const T *__restrict__ dP, const float *__restrict__ rowdot,
                                                                  T *__restrict__ dk, T *__restrict__ dv, int L, int H, float scaling)
{
    pdl_wait();
    extern __shared__ __align__(16) float att_smem[];
    const int Lp = L + 1, head = blockIdx.y, k0 = blockIdx.x * ATT_TQ, nk = min(ATT_TQ, L - k0);
    float *p_tile = att_smem, *ds_tile = att_smem + ATT_TQ * Lp;        // [key][query]
    const size_t hoff = (size_t)head * H * L;
    const bool vec = nk == ATT_TQ && L % 4 == 0 && (((uintptr_t)P | (uintptr_t)dP) & (4 * sizeof(T) - 1)) == 0;
    for (int query = threadIdx.x; query < L; query += ATT_THREADS) {
        const size_t off = ((size_t)head * L + query) * L + k0;
        const float dot = rowdot[(size_t)head * L + query];
        float p[ATT_TQ], g[ATT_TQ];
        if (vec) { ld4(P + off, p); ld4(dP + off, g); }
        else {
#pragma unroll
            for (int kk = 0; kk < ATT_TQ; kk++) { p[kk] = ld0(kk < nk, P + off + kk); g[kk] = ld0(kk < nk, dP + off + kk); }
        }
#pragma unroll
        for (int kk = 0; kk < ATT_TQ; kk++) { p_tile[kk * Lp + query] = p[kk]; ds_tile[kk * Lp + query] = __fmul_rn(__fsub_rn(g[kk], dot), p[kk]); }
    }
    __syncthreads();
    rows_times_tile(datt + hoff, p_tile, Lp, H, L, dv + hoff, k0, nk, 1.0f);
    rows_times_tile(q + hoff, ds_tile, Lp, H, L, dk + hoff, k0, nk, scaling);
}

// ---------------------------------------------------------------- the same three kernels on mma.sync
// For half precision: sixteen queries (keys) per CTA, every product as m16n8k8 TF32 instructions, some 40 instructions for 4096
// multiply-adds where the kernels above take 220, and a quarter of what they fetch from L2.  fp16 values are TF32 values; the fp32
// tile of probabilities (or dS) is split into two TF32 parts, both rounded to nearest (|x - hi - lo| <= 2^-23 |x|, small term first).  The accumulation
// of mma.sync truncates, so that chains are short: the sums of four k-steps of scores, of two k-steps of both parts of a tile are added
// to fp32 registers with ordinary rounding.  Of 262 144 dq and dk (4 heads x 512 x 64) 130 are not the half nearest to the 64-bit value, of the
// kernels above 146; with four k-steps a chain and the low part cut off they were 228.  (fp32 operands, split the same way, gave
// three times the FFMA kernels' error against 64 bits, 2.2e-7 against 7.5e-8, so they stay there.)
//   scores:        A = the sixteen columns in shared memory, B = rows of M straight from memory (each is used by one warp only)
//   rows of M x tile: A = rows of M from memory, four neighbouring tokens per lane (the order of k within a step is free as long as
//                  both operands follow it), B = the tile; warps that the rows leave over share the tokens
// Where they pay, with both sides measured: am_threads.
static constexpr int AM_Q = 16, AM_AP = 24;       // queries per CTA; pitch of a row of the column tile (conflict-free fragments)
__host__ __device__ inline int am_pitch(int L) { return ((L + 31) & ~31) + 16; }       // floats of a tile row: eight rows by four lanes of 16 bytes hit all banks
struct AmSplit { int mt, js; };                   // blocks of sixteen rows side by side, shares of the tokens
__host__ __device__ inline AmSplit am_split(int L, int H, int NW)
{
    AmSplit s;
    const int blocks = (H + 15) / 16, steps = (L + 15) / 16;
    s.mt = blocks < NW ? blocks : NW;
    s.js = NW / s.mt < steps ? NW / s.mt : steps;
    return s;
}
__device__ __forceinline__ void am_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// four neighbours, zero at or past `left`
__device__ __forceinline__ void am_ld4(const __half *p, int left, bool vec, float (&v)[4])
{
    if (vec && left >= 4) { ld4(p, v); return; }
#pragma unroll
    for (int i = 0; i < 4; i++) v[i] = ld0(i < left, p + i);
}

// tile[row][j] = alpha * sum_d cols[d][row] M[d][j] for the sixteen rows and j < L, zero for L <= j < the next multiple of 16
template <int NT>
__device__ __forceinline__ void am_scores(const float *cols, const __half *__restrict__ M, float *tile, int Lp, int H, int L, float alpha)
{
    constexpr int NW = NT / 32, NTL = NT == 512 ? 2 : 4, KB = 4;            // 8-key tiles of a warp side by side; k-steps whose loads are in flight
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    for (int n0 = warp * 8 * NTL; n0 < ((L + 15) & ~15); n0 += NW * 8 * NTL) {
        float acc[NTL][4];
#pragma unroll
        for (int i = 0; i < NTL; i++)
#pragma unroll
            for (int q = 0; q < 4; q++) acc[i][q] = 0.f;
        for (int d0 = 0; d0 < H; d0 += 8 * KB) {
            float m[KB][NTL][2], tmp[NTL][4];
#pragma unroll
            for (int u = 0; u < KB; u++)
#pragma unroll
                for (int i = 0; i < NTL; i++)
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const int d = d0 + 8 * u + t + 4 * h, n = n0 + 8 * i + g;
                        m[u][i][h] = ld0(d < H && n < L, M + (size_t)d * L + n);
                    }
#pragma unroll
            for (int i = 0; i < NTL; i++)
#pragma unroll
                for (int q = 0; q < 4; q++) tmp[i][q] = 0.f;
#pragma unroll
            for (int u = 0; u < KB; u++) {
                if (d0 + 8 * u >= H) break;
                const float *c = cols + (d0 + 8 * u + t) * AM_AP + g;
                const uint32_t a4[4] = {__float_as_uint(c[0]), __float_as_uint(c[8]), __float_as_uint(c[4 * AM_AP]), __float_as_uint(c[4 * AM_AP + 8])};
#pragma unroll
                for (int i = 0; i < NTL; i++) am_mma(tmp[i], a4, __float_as_uint(m[u][i][0]), __float_as_uint(m[u][i][1]));
            }
#pragma unroll
            for (int i = 0; i < NTL; i++)
#pragma unroll
                for (int q = 0; q < 4; q++) acc[i][q] += tmp[i][q];
        }
#pragma unroll
        for (int i = 0; i < NTL; i++) {
            const int n = n0 + 8 * i + 2 * t;
            if (n >= ((L + 15) & ~15)) break;
            *reinterpret_cast<float2 *>(tile + g * Lp + n) = make_float2(__fmul_rn(acc[i][0], alpha), __fmul_rn(acc[i][1], alpha));
            *reinterpret_cast<float2 *>(tile + (g + 8) * Lp + n) = make_float2(__fmul_rn(acc[i][2], alpha), __fmul_rn(acc[i][3], alpha));
        }
    }
}

// out[d][t0 + n] = alpha * sum_j M[d][j] tile[n][j]  for d < H, n < nt.  share: [js][rows of a pass][16], added in order.
template <int NT>
__device__ __forceinline__ void am_rows(const __half *__restrict__ M, const float *tile, int Lp, int H, int L, __half *__restrict__ out, int t0, int nt, float alpha, float *share, AmSplit sp)
{
    constexpr int U = 2;                                                   // steps of 16 tokens whose loads are in flight
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3, jp = warp / sp.mt, wr = warp - jp * sp.mt;
    const int steps = (L + 15) / 16, per = (steps + sp.js - 1) / sp.js, s0 = jp * per, s1 = min(steps, s0 + per);
    const bool vec = L % 4 == 0 && (reinterpret_cast<uintptr_t>(M) & (4 * sizeof(__half) - 1)) == 0;
    for (int pass = 0; pass < H; pass += 16 * sp.mt) {
        const int d0 = pass + 16 * wr;
        float acc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
        if (jp < sp.js && d0 < H) {
            const __half *r0 = M + (size_t)min(d0 + g, H - 1) * L + 4 * t, *r1 = M + (size_t)min(d0 + g + 8, H - 1) * L + 4 * t;
            const float *b0 = tile + g * Lp + 4 * t, *b1 = b0 + 8 * Lp;
            for (int s = s0; s < s1; s += U) {
                float m[U][2][4];
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const int left = s + u < s1 ? L - 16 * (s + u) - 4 * t : 0;
                    am_ld4(r0 + 16 * (s + u), left, vec, m[u][0]);
                    am_ld4(r1 + 16 * (s + u), left, vec, m[u][1]);
                }
#pragma unroll
                for (int u = 0; u < U; u++) {
                    if (s + u >= s1) break;
                    float bv[2][4], tmp[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
                    uint32_t a4[2][4], bh[2][4], bl[2][4];
                    *reinterpret_cast<float4 *>(bv[0]) = *reinterpret_cast<const float4 *>(b0 + 16 * (s + u));
                    *reinterpret_cast<float4 *>(bv[1]) = *reinterpret_cast<const float4 *>(b1 + 16 * (s + u));
#pragma unroll
                    for (int h = 0; h < 2; h++)                            // tokens 4 t + 2 h and 4 t + 2 h + 1 are k = t and t + 4
#pragma unroll
                        for (int q = 0; q < 4; q++) a4[h][q] = __float_as_uint(m[u][q & 1][2 * h + (q >> 1)]);
#pragma unroll
                    for (int n = 0; n < 2; n++)
#pragma unroll
                        for (int q = 0; q < 4; q++) tc::split_tf32_rn(bv[n][q], bh[n][q], bl[n][q]);
#pragma unroll
                    for (int part = 0; part < 2; part++)
#pragma unroll
                        for (int h = 0; h < 2; h++)
#pragma unroll
                            for (int n = 0; n < 2; n++) am_mma(tmp[n], a4[h], part ? bh[n][2 * h] : bl[n][2 * h], part ? bh[n][2 * h + 1] : bl[n][2 * h + 1]);
#pragma unroll
                    for (int n = 0; n < 2; n++)
#pragma unroll
                        for (int q = 0; q < 4; q++) acc[n][q] += tmp[n][q];
                }
            }
            if (sp.js > 1) {
#pragma unroll
                for (int n = 0; n < 2; n++)
#pragma unroll
                    for (int q = 0; q < 4; q++) share[((jp * sp.mt + wr) * 16 + g + 8 * (q >> 1)) * 16 + 8 * n + 2 * t + (q & 1)] = acc[n][q];
            } else {
#pragma unroll
                for (int n = 0; n < 2; n++)
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        const int d = d0 + g + 8 * (q >> 1), c = 8 * n + 2 * t + (q & 1);
                        if (d < H && c < nt) st(out + (size_t)d * L + t0 + c, __fmul_rn(acc[n][q], alpha));
                    }
            }
        }
        if (sp.js > 1) {
            __syncthreads();
            for (int e = threadIdx.x; e < sp.mt * 256; e += NT) {
                const int d = pass + (e >> 4), c = e & 15;
                if (d >= H || c >= nt) continue;
                float sum = share[e];
                for (int p = 1; p < sp.js; p++) sum += share[p * sp.mt * 256 + e];
                st(out + (size_t)d * L + t0 + c, __fmul_rn(sum, alpha));
            }
            __syncthreads();
        }
    }
}
// cols[d][i] = A[d][t0 + i], zero past the last token and for d past H up to a multiple of 32
template <int NT> __device__ __forceinline__ void am_columns(const __half *__restrict__ A, float *cols, int H, int L, int t0)
{
    for (int i = threadIdx.x; i < ((H + 31) & ~31) * AM_Q; i += NT) {
        const int d = i / AM_Q, c = i % AM_Q;
        cols[d * AM_AP + c] = ld0(d < H && t0 + c < L, A + (size_t)d * L + t0 + c);
    }
}

template <int NT>
__global__ void __launch_bounds__(NT) mma_attn_fw_kernel(const __half *__restrict__ q, const __half *__restrict__ k, const __half *__restrict__ v,
                                                         __half *__restrict__ P, __half *__restrict__ att, int L, int H, float scaling)
{
    pdl_wait();
    extern __shared__ __align__(16) float att_smem[];
    const int Lp = am_pitch(L), head = blockIdx.y, t0 = blockIdx.x * AM_Q, nt = min(AM_Q, L - t0);
    float *tile = att_smem, *cols = tile + AM_Q * Lp, *share = cols + ((H + 31) & ~31) * AM_AP;
    const size_t hoff = (size_t)head * H * L;
    am_columns<NT>(q + hoff, cols, H, L, t0);
    __syncthreads();
    am_scores<NT>(cols, k + hoff, tile, Lp, H, L, scaling);
    __syncthreads();
    // row softmax, a warp per query: max, Schraudolph exp of (x - max), divide by the row sum  [ref: pulp_act_fp32.c:187-245]
    const int lane = threadIdx.x & 31;
    for (int t = threadIdx.x >> 5; t < nt; t += NT / 32) {
        float *row = tile + t * Lp;
        float m = -FLT_MAX;
        for (int j = lane; j < L; j += 32) m = fmaxf(m, row[j]);
        m = warp_max(m);
        float s = 0.f;
        for (int j = lane; j < L; j += 32) { const float e = fastexp_gist_dev(__fsub_rn(row[j], m)); row[j] = e; s += e; }
        s = warp_sum(s);
        __half *prow = P + ((size_t)head * L + t0 + t) * L;
        for (int j = lane; j < L; j += 32) { const float p = __fdiv_rn(row[j], s); row[j] = p; st(prow + j, p); }
    }
    __syncthreads();
    am_rows<NT>(v + hoff, tile, Lp, H, L, att + hoff, t0, nt, 1.0f, share, am_split(L, H, NT / 32));
}

// Query-tiled half of the backward pass: dP (written), row sums of dP * P (written), dq (written).
template <int NT>
__global__ void __launch_bounds__(NT) mma_attn_bw_query_kernel(const __half *__restrict__ datt, const __half *__restrict__ v, const __half *__restrict__ k,
                                                               const __half *__restrict__ P, __half *__restrict__ dP, float *__restrict__ rowdot,
                                                               __half *__restrict__ dq, int L, int H, float scaling)
{
    pdl_wait();
    extern __shared__ __align__(16) float att_smem[];
    const int Lp = am_pitch(L), head = blockIdx.y, t0 = blockIdx.x * AM_Q, nt = min(AM_Q, L - t0);
    float *tile = att_smem, *cols = tile + AM_Q * Lp, *share = cols + ((H + 31) & ~31) * AM_AP;
    const size_t hoff = (size_t)head * H * L;
    am_columns<NT>(datt + hoff, cols, H, L, t0);
    __syncthreads();
    am_scores<NT>(cols, v + hoff, tile, Lp, H, L, 1.0f);
    __syncthreads();
    const int lane = threadIdx.x & 31;
    for (int t = threadIdx.x >> 5; t < nt; t += NT / 32) {
        // dS = (dP - sum_key dP P) P   [ref: lib/sources/pulp_act_fp32.c:335-392]
        float *row = tile + t * Lp;
        const size_t roff = ((size_t)head * L + t0 + t) * L;
        float s = 0.f;
        for (int j0 = 0; j0 < L; j0 += 256) {
            float p[8];
#pragma unroll
            for (int u = 0; u < 8; u++) p[u] = ld0(j0 + 32 * u + lane < L, P + roff + j0 + 32 * u + lane);
#pragma unroll
            for (int u = 0; u < 8; u++) {
                const int j = j0 + 32 * u + lane;
                if (j >= L) break;
                float d = row[j];
                d = __half2float(__float2half_rn(d)); row[j] = d;          // the value the caller sees in dP
                st(dP + roff + j, d);
                s = fmaf(d, p[u], s);
            }
        }
        s = warp_sum(s);
        if (lane == 0) rowdot[(size_t)head * L + t0 + t] = s;
        for (int j0 = 0; j0 < L; j0 += 256) {
            float p[8];
#pragma unroll
            for (int u = 0; u < 8; u++) p[u] = ld0(j0 + 32 * u + lane < L, P + roff + j0 + 32 * u + lane);
#pragma unroll
            for (int u = 0; u < 8; u++) {
                const int j = j0 + 32 * u + lane;
                if (j < L) row[j] = __fmul_rn(__fsub_rn(row[j], s), p[u]);
            }
        }
    }
    __syncthreads();
    am_rows<NT>(k + hoff, tile, Lp, H, L, dq + hoff, t0, nt, scaling, share, am_split(L, H, NT / 32));
}

// Key-tiled half: columns of P and of dS = (dP - rowdot) P for sixteen keys against all queries, then
// dv[d][key] = sum_query datt[d][query] P[query][key] and dk[d][key] = scaling * sum_query q[d][query] dS[query][key].
template <int NT>
__global__ void __launch_bounds__(NT) mma_attn_bw_key_kernel(const __half *__restrict__ datt, const __half *__restrict__ q, const __half *__restrict__ P,
                                                             const __half *__restrict__ dP, const float *__restrict__ rowdot,
                                                             __half *__restrict__ dk, __half *__restrict__ dv, int L, int H, float scaling)
{
    pdl_wait();
    extern __shared__ __align__(16) float att_smem[];
    const int Lp = am_pitch(L), head = blockIdx.y, k0 = blockIdx.x * AM_Q, nk = min(AM_Q, L - k0);
    float *p_tile = att_smem, *ds_tile = p_tile + AM_Q * Lp, *share = ds_tile + AM_Q * Lp;        // [key][query]
    const size_t hoff = (size_t)head * H * L;
    const bool vec = L % 4 == 0 && (((uintptr_t)P | (uintptr_t)dP) & (4 * sizeof(__half) - 1)) == 0;
    const int queries = (L + 15) & ~15;                                    // zero beyond the last one
    for (int e = threadIdx.x; e < queries * 4; e += NT) {
        const int query = e >> 2, c = (e & 3) * 4, left = query < L ? nk - c : 0;
        const size_t off = ((size_t)head * L + min(query, L - 1)) * L + k0 + c;
        const float dot = rowdot[(size_t)head * L + min(query, L - 1)];
        float p[4], d[4];
        am_ld4(P + off, left, vec, p);
        am_ld4(dP + off, left, vec, d);
#pragma unroll
        for (int i = 0; i < 4; i++) { p_tile[(c + i) * Lp + query] = p[i]; ds_tile[(c + i) * Lp + query] = i < left ? __fmul_rn(__fsub_rn(d[i], dot), p[i]) : 0.f; }
    }
    __syncthreads();
    const AmSplit sp = am_split(L, H, NT / 32);
    am_rows<NT>(datt + hoff, p_tile, Lp, H, L, dv + hoff, k0, nk, 1.0f, share, sp);
    am_rows<NT>(q + hoff, ds_tile, Lp, H, L, dk + hoff, k0, nk, scaling, share, sp);
}

// ---------------------------------------------------------------- host side
static size_t attn_smem_bytes(int L, int H, int tiles) { return ((size_t)H * ATT_TQ + (size_t)tiles * ATT_TQ * (L + 1)) * sizeof(float); }
static size_t am_smem_bytes(int L, int H, int tiles, int NT)
{
    const AmSplit sp = am_split(L, H, NT / 32);
    return ((size_t)tiles * AM_Q * am_pitch(L) + (tiles == 1 ? (size_t)((H + 31) & ~31) * AM_AP : 0) + (sp.js > 1 ? (size_t)sp.js * sp.mt * 256 : 0)) * sizeof(float);
}
static const size_t AM_SMEM_MAX = 200 * 1024;

// True when the fused kernels take this shape: the tiles of one CTA must fit in shared memory.
bool attn_fused_ok(int L, int H)
{
    return L >= 1 && H >= 1 && attn_smem_bytes(L, H, 2) <= 200 * 1024;
}
// Threads of the kernels with sixteen queries per CTA, 0: four queries on FFMA.  The former win where that leaves enough CTAs; sixteen warps
// each where there is no more than one CTA per SM.  (us, four queries / sixteen: 8 heads x 459 tokens x 16 (232 CTAs) 23.9 / 16.3
// forward, 26.1 / 15.6 and 21.2 / 15.4 backward; 4 x 500 x 64 (128) 33.3 / 19.7 (with eight warps 35.5), 40.9 / 16.7, 25.7 / 16.1; 8 x
// 330 x 64 (168) 41.0 / 30.3, 39.4 / 28.8, 27.0 / 24.8; with few CTAs their longer chain costs more: 4 x 39 x 16 (12) 4.6 / 6.0, 4.7 / 5.8,
// 3.2 / 4.6; 4 x 129 x 32 (36) 7.3 / 7.5, 6.6 / 7.0, 4.7 / 6.9.)
template <class T> static int am_threads(int L, int H, int heads)
{
    const long long ctas = (long long)ceil_div(L, AM_Q) * heads;
    const int NT = ctas <= sm_count() ? 512 : 256;
    return sizeof(T) == 2 && ctas >= 96 && am_smem_bytes(L, H, 1, NT) <= AM_SMEM_MAX && am_smem_bytes(L, H, 2, NT) <= AM_SMEM_MAX ? NT : 0;
}
// (the default without asking is 48 KB)
template <class K> static void am_allow(K kernel, size_t smem) { if (smem > 48 * 1024) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); }

template <class T>
void attn_fw(const T *q, const T *k, const T *v, T *P, T *att, int L, int H, int heads, float scaling)
{
    if constexpr (sizeof(T) == 2)
        if (const int NT = am_threads<T>(L, H, heads)) {
            const size_t smem = am_smem_bytes(L, H, 1, NT);
            const dim3 grid(ceil_div(L, AM_Q), heads);
            if (NT == 512) { am_allow(mma_attn_fw_kernel<512>, smem); TL_LAUNCH(mma_attn_fw_kernel<512>, grid, 512, smem, q, k, v, P, att, L, H, scaling); }
            else { am_allow(mma_attn_fw_kernel<256>, smem); TL_LAUNCH(mma_attn_fw_kernel<256>, grid, 256, smem, q, k, v, P, att, L, H, scaling); }
            return;
        }
    const size_t smem = attn_smem_bytes(L, H, 1);
    am_allow(attn_fw_kernel<T>, smem);
    TL_LAUNCH((attn_fw_kernel<T>), dim3(ceil_div(L, ATT_TQ), heads), ATT_THREADS, smem, q, k, v, P, att, L, H, scaling);
}

template <class T>
void attn_bw(const T *datt, const T *q, const T *k, const T *v, const T *P, T *dP, float *rowdot, T *dq, T *dk, T *dv,
             int L, int H, int heads, float scaling)
{
    if constexpr (sizeof(T) == 2)
        if (const int NT = am_threads<T>(L, H, heads)) {
            const size_t smem1 = am_smem_bytes(L, H, 1, NT), smem2 = am_smem_bytes(L, H, 2, NT);
            const dim3 grid(ceil_div(L, AM_Q), heads);
            if (NT == 512) {
                am_allow(mma_attn_bw_query_kernel<512>, smem1); am_allow(mma_attn_bw_key_kernel<512>, smem2);
                TL_LAUNCH(mma_attn_bw_query_kernel<512>, grid, 512, smem1, datt, v, k, P, dP, rowdot, dq, L, H, scaling);
                TL_LAUNCH(mma_attn_bw_key_kernel<512>, grid, 512, smem2, datt, q, P, dP, rowdot, dk, dv, L, H, scaling);
            } else {
                am_allow(mma_attn_bw_query_kernel<256>, smem1); am_allow(mma_attn_bw_key_kernel<256>, smem2);
                TL_LAUNCH(mma_attn_bw_query_kernel<256>, grid, 256, smem1, datt, v, k, P, dP, rowdot, dq, L, H, scaling);
                TL_LAUNCH(mma_attn_bw_key_kernel<256>, grid, 256, smem2, datt, q, P, dP, rowdot, dk, dv, L, H, scaling);
            }
            return;
        }
    const size_t smem1 = attn_smem_bytes(L, H, 1), smem2 = attn_smem_bytes(L, 0, 2);
    am_allow(attn_bw_query_kernel<T>, smem1); am_allow(attn_bw_key_kernel<T>, smem2);
    const dim3 grid(ceil_div(L, ATT_TQ), heads);
    TL_LAUNCH((attn_bw_query_kernel<T>), grid, ATT_THREADS, smem1, datt, v, k, P, dP, rowdot, dq, L, H, scaling);
    TL_LAUNCH((attn_bw_key_kernel<T>), grid, ATT_THREADS, smem2, datt, q, P, dP, rowdot, dk, dv, L, H, scaling);
}

#define INST(T)                                                                                                        \
    template void attn_fw<T>(const T *, const T *, const T *, T *, T *, int, int, int, float);                        \
    template void attn_bw<T>(const T *, const T *, const T *, const T *, const T *, T *, float *, T *, T *, T *, int, int, int, float);
INST(float)
INST(__half)

} // namespace tl

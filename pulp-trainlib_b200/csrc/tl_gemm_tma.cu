// TMA-fed tensor-core GEMM for the large products of the `mm` family
// [ref: lib/sources/pulp_matmul_fp32.c:190-262, lib/sources/pulp_matmul_fp16.c:191-262]:
//     C[N x M] = alpha * A[N x K] * B[K x M] (+ bias) (+ C)
//
// Kernel: persistent CTAs walk 128 x BN tiles of C (rows of tiles in groups of eight, so that a group's operands stay in L2).
// A producer warp issues cp.async.bulk.tensor (128-byte swizzle; out-of-range rows and k read as zero, so no tail code) into
// a ring of shared-memory stages and runs ahead across tiles; an issuer warp runs tcgen05.mma from shared-memory descriptors
// into tensor memory and releases each stage with tcgen05.commit; four warps read finished accumulators with tcgen05.ld and
// write C (any strides).  What bounds single CTAs is the way from L2 into the SM: 48 KB per 512 tensor cycles of a 128 x 256 fp16 tile.
//   PAIR: two CTAs share a 256 x BN tile (cta_group::2): each holds its 128 rows of A and half of B's rows, 32 KB instead of 48.
//         fp16 4096^3 so: tensor pipe active 89 % of the cycles, 102 us at the 1.25 GHz that the power limit leaves it.
//   fp16: kind::f16, operands in place whichever index is contiguous: K-major tiles ([row][64 k]) or MN-major ones ([k][64 rows],
//         the majorness bits of the instruction descriptor).  Packing B of a plain product into K-major scratch took 43 of the
//         155 us of a 4096^3 product.  BN = 256 with two accumulators: a tile's epilogue runs under the next tile's products.
//   fp32: 3xTF32 on packed (hi, lo) pairs.  B_hi and B_lo lie behind each other: D0 += A_hi [B_hi | B_lo]^T is one instruction of
//         N = 2 BN (A_hi is read once), D1 += A_lo B_hi^T a second one; the epilogue adds the three parts, whose accumulation
//         chains are a third as long as one common chain (the accumulator truncates).
// Measured, whole call: fp16 4096^3 173 -> 120 us over seconds (101 us in short runs), fp16 2048^3 29 -> 17.5 us, fp32 2048^3 118 -> 89 us, fp32 1000 x 600 x 1300
// (B transposed) 31 -> 20.3 us, fp32 300 x 2050 x 914 67 -> 26 us.
// Few tiles: `splits` CTAs share the K steps of a tile and write partial tiles; tm_reduce_kernel adds them in order.  A contraction
// may run over several segments (the streams of a batch), which the tensor maps' third index selects, as it selects a batch.
// No multicast loads.  Every wait is bounded and reports through the status word.
#include "tl_kernels.h"
#include "tl_tc.cuh"
#include <algorithm>

namespace tl {

using namespace tc;

int *tc_status_word();          // tl_conv_tc.cu
void *tc_encode_tiled_fn();     // tl_conv_tc.cu: cuTensorMapEncodeTiled through the runtime's driver entry point query

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                  const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static constexpr int TM_BM = 128;
static constexpr int TM_THREADS = 192;          // warps 0-3: epilogue, warp 4: TMA producer, warp 5: MMA issuer
static constexpr int TM_MAX_STAGES = 8;
static constexpr uint32_t TM_RING = 200 * 1024;

template <class T> struct TmCfg;
template <> struct TmCfg<__half> { static constexpr int BK = 64, PARTS = 1; };
template <> struct TmCfg<float>  { static constexpr int BK = 32, PARTS = 2; };

struct TmParams {
    void *C; const void *bias; float *part;
    int N, M, K;
    long long c_rs, c_cs, c_bs;
    float alpha; int accumulate, bias_mode;
    int BN, tiles_m, tiles_n, tiles, ksteps, kps, splits, stages, pair, a_mn, b_mn, b_one;      // b_one: all products of a batch share B
    uint32_t stage_bytes;
    int *status;
};

__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap *m, uint64_t *bar, int x, int y, int z)
{
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
                 ::"r"(dst), "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z) : "memory");
}
// The same for a CTA pair: the barrier (a cluster address) may be the other CTA's.
__device__ __forceinline__ void tma_load_3d_pair(uint32_t dst, const CUtensorMap *m, uint32_t bar, int x, int y, int z)
{
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%3, %4, %5}], [%2];"
                 ::"r"(dst), "l"(reinterpret_cast<uint64_t>(m)), "r"(bar), "r"(x), "r"(y), "r"(z) : "memory");
}
// One MMA; PAIR: 256 rows, 128 in each CTA of the pair, and half of B's rows from each CTA's shared memory.
template <bool HALF, bool PAIR> __device__ __forceinline__ void tm_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc)
{
    if constexpr (!PAIR) { if constexpr (HALF) mma_f16_ss(d, a, b, idesc, acc); else mma_tf32_ss(d, a, b, idesc, acc); }
    else if constexpr (HALF)
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                     ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(acc) : "memory");
    else
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::2.kind::tf32 [%0], %1, %2, %3, p;\n\t}"
                     ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(acc) : "memory");
}
// An arrival on the barrier (PAIR: of both CTAs) when the MMAs issued so far have completed.
template <bool PAIR> __device__ __forceinline__ void tm_commit(uint64_t *bar)
{
    if constexpr (!PAIR) mma_commit(bar);
    else asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)), "h"((uint16_t)3) : "memory");
}
__device__ __forceinline__ uint32_t tm_mapa(uint32_t addr, uint32_t rank)
{
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
    return a;
}
__device__ __forceinline__ void tm_arrive_at(uint32_t bar)           // a cluster address
{
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Bounded wait (about a second): polls back to back, or `nap` ns apart.
__device__ __forceinline__ bool tm_wait(uint64_t *bar, uint32_t parity, volatile int *failed, uint32_t nap = 0)
{
    for (uint32_t i = 0; i < 20000000u; i++) {
        if (mbar_try_wait(bar, parity)) return true;
        if (nap) __nanosleep(nap);
        if ((i & 63u) == 63u && *failed) return false;
    }
    *failed = 1;
    return false;
}
__device__ __forceinline__ void tm_cluster_sync()
{
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
// four neighbouring results of one row: alpha, bias, accumulate, store
template <class T> __device__ __forceinline__ void tm_store4(const TmParams &p, T *crow, int row, int col, const float (&in)[4], bool vec)
{
    const T *bias = reinterpret_cast<const T *>(p.bias);
    const int live = min(4, p.M - col);
    float r[4];
    const float brow = ld0(p.bias_mode == 1, bias + row);
#pragma unroll
    for (int q = 0; q < 4; q++) {
        r[q] = p.alpha * in[q] + brow;
        if (p.bias_mode == 2 && q < live) r[q] += ld(bias + col + q);
    }
    T *dst = crow + (long long)col * p.c_cs;
    if (vec && live == 4) {
        if constexpr (sizeof(T) == 2) {
            const __half2 a = __floats2half2_rn(r[0], r[1]), b = __floats2half2_rn(r[2], r[3]);
            *reinterpret_cast<uint2 *>(dst) = make_uint2(*reinterpret_cast<const uint32_t *>(&a), *reinterpret_cast<const uint32_t *>(&b));
        } else *reinterpret_cast<float4 *>(dst) = make_float4(r[0], r[1], r[2], r[3]);
    } else {
#pragma unroll
        for (int q = 0; q < 4; q++) if (q < live) { T *o = dst + q * p.c_cs; st(o, p.accumulate ? r[q] + ld(o) : r[q]); }
    }
}

// tile -> (batch, row block, column block): eight row blocks share a sweep over the columns
__device__ __forceinline__ void tm_locate(const TmParams &p, int tile, int &b, int &rb, int &cb)
{
    const int per = p.tiles_m * p.tiles_n;
    b = tile / per;
    const int t = tile - b * per, g = t / (8 * p.tiles_m), in = t - g * 8 * p.tiles_m, rows = min(8, p.tiles_n - 8 * g);
    rb = 8 * g + in % rows; cb = in / rows;
}

// maps: a0 = A (hi), a1 = A lo (fp32 only), b0 = B (hi), b1 = B lo
template <class T, bool PAIR>
__global__ void __launch_bounds__(TM_THREADS) gemm_tma_kernel(const __grid_constant__ CUtensorMap a0, const __grid_constant__ CUtensorMap a1,
                                                              const __grid_constant__ CUtensorMap b0, const __grid_constant__ CUtensorMap b1, const __grid_constant__ TmParams p)
{
    pdl_wait();
    typedef TmCfg<T> Cfg;
    constexpr int BK = Cfg::BK;
    constexpr bool HALF = sizeof(T) == 2;
    constexpr uint32_t A_BYTES = TM_BM * 128u;                                      // one 128-byte row per tile row (or 64 k of 128 rows)
    extern __shared__ unsigned char tsm_raw[];
    const uint32_t sbase = (smem_u32(tsm_raw) + 1023u) & ~1023u;                    // swizzle atoms want 1024-byte alignment
    __shared__ uint64_t full[TM_MAX_STAGES], empty[TM_MAX_STAGES], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_slot;
    __shared__ int failed_s;
    volatile int *failed = &failed_s;

    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;       // (a warp number the compiler knows to be uniform)
    const int BN = p.BN, ST = p.stages, nbuf = HALF ? 2 : 1;
    const int BNL = PAIR ? BN / 2 : BN;                                             // rows of B in this CTA's shared memory
    const uint32_t B_BYTES = (uint32_t)BNL * 128u;
    const int group = PAIR ? 2 : p.splits, rank = (int)blockIdx.x % group, first = (int)blockIdx.x / group, step = (int)gridDim.x / group;
    const int ks0 = PAIR ? 0 : p.ksteps * rank / p.splits, ks1 = PAIR ? p.ksteps : p.ksteps * (rank + 1) / p.splits;
    constexpr int ROWS = PAIR ? 2 * TM_BM : TM_BM;
    const int row_of_tile = PAIR ? rank * TM_BM : 0;

    if (tid == 0) {
        for (int s = 0; s < ST; s++) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        for (int b = 0; b < 2; b++) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], PAIR ? 8 : 4); }
        failed_s = 0;
        fence_barrier_init();
        tma_prefetch_desc(&a0); tma_prefetch_desc(&b0);
        if (!HALF) { tma_prefetch_desc(&a1); tma_prefetch_desc(&b1); }
    }
    if (warp == 0) {
        if constexpr (PAIR) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&tmem_slot)) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else { tmem_alloc(&tmem_slot, 512); tmem_relinquish(); }
    }
    tc_fence_before();
    if constexpr (PAIR) tm_cluster_sync();                                          // the other CTA's barriers are initialised too
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    // The producer and the issuers run their loops as whole warps and elect a thread only around the instructions themselves:
    // operands of tcgen05.mma are uniform registers, and in a branch on lane 0 every one of them costs a detour (a 4096^3 fp16
    // product took 177 us that way and 129 us this way, before pairs).
    if (warp == 4) {
        const uint32_t full0 = PAIR ? tm_mapa(smem_u32(&full[0]), 0) : 0u;             // the pair's leader counts both CTAs' bytes
        int s = 0;
        uint32_t phase = 1;                                                         // the first pass over the ring finds it empty
        bool ok = true;
        for (int tile = first; tile < p.tiles && ok; tile += step) {
            int b, rb, cb;
            tm_locate(p, tile, b, rb, cb);
            const int row0 = rb * ROWS + row_of_tile, col0 = cb * BN + (PAIR ? rank * BNL : 0);
            int seg = ks0 / p.kps, kt = ks0 - seg * p.kps;                          // segment of the contraction, K step inside it
            for (int k = ks0; k < ks1; k++) {
                const int za = b + seg, zb = (p.b_one ? 0 : b) + seg;
                if (!tm_wait(&empty[s], phase, failed)) { ok = false; break; }
                if (elect_one()) {
                    const uint32_t st = sbase + s * p.stage_bytes, sb = st + Cfg::PARTS * A_BYTES;
                    const uint32_t bar = full0 + 8u * s;
                    auto load = [&](uint32_t dst, const CUtensorMap *m, int x, int y, int z) {
                        if constexpr (PAIR) tma_load_3d_pair(dst, m, bar, x, y, z);
                        else tma_load_3d(dst, m, &full[s], x, y, z);
                    };
                    if (!PAIR || rank == 0) mbar_arrive_expect_tx(&full[s], PAIR ? 2 * p.stage_bytes : p.stage_bytes);
                    if (HALF && p.a_mn) { for (int j = 0; j < 2; j++) load(st + j * 8192u, &a0, row0 + 64 * j, kt * BK, za); }
                    else load(st, &a0, kt * BK, row0, za);
                    if (!HALF) load(st + A_BYTES, &a1, kt * BK, row0, za);
                    if (HALF && p.b_mn) { for (int j = 0; j < BNL / 64; j++) load(sb + j * 8192u, &b0, col0 + 64 * j, kt * BK, zb); }
                    else load(sb, &b0, kt * BK, col0, zb);
                    if (!HALF) load(sb + B_BYTES, &b1, kt * BK, col0, zb);
                }
                __syncwarp();
                if (++kt == p.kps) { kt = 0; seg++; }
                if (++s == ST) { s = 0; phase ^= 1u; }
            }
        }
    } else if (warp >= 5) {
        if (!PAIR || rank == 0) {
            const uint32_t majors = (p.a_mn ? IDESC_A_MN_MAJOR : 0u) | (p.b_mn ? IDESC_B_MN_MAJOR : 0u);
            const uint32_t idesc = HALF ? (mma_idesc(FMT_F16, ROWS, BN) | majors) : mma_idesc(FMT_TF32, ROWS, 2 * BN), idesc_lo = mma_idesc(FMT_TF32, ROWS, BN);
            // descriptor words that do not depend on the stage, and the step of one MMA (32 bytes or 16 rows of K) in 16-byte units
            const uint64_t desc_a = p.a_mn ? smem_desc_swizzled(0, 8192u, 1024u, LAYOUT_SW128) : smem_desc_kmajor_sw128(0, 1024);
            const uint64_t desc_b = p.b_mn ? smem_desc_swizzled(0, 8192u, 1024u, LAYOUT_SW128) : smem_desc_kmajor_sw128(0, 1024);
            const uint32_t step_a = p.a_mn ? 128u : 2u, step_b = p.b_mn ? 128u : 2u;
            int s = 0, tl = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int tile = first; tile < p.tiles && ok; tile += step, tl++) {
                const int buf = tl % nbuf, use_b = tl / nbuf;
                if (use_b > 0 && !tm_wait(&acc_empty[buf], (uint32_t)(use_b - 1) & 1u, failed)) { ok = false; break; }
                tc_fence_after();
                const uint32_t d = tmem + (HALF ? buf * 256 : 0);
                uint32_t acc = 0;
                for (int kt = ks0; kt < ks1; kt++) {
                    if (!tm_wait(&full[s], phase, failed)) { ok = false; break; }
                    tc_fence_after();
                    if (elect_one()) {
                        const uint32_t st = sbase + s * p.stage_bytes, sb = st + Cfg::PARTS * A_BYTES;
                        const uint64_t da = desc_a + (st >> 4), db = desc_b + (sb >> 4);
#pragma unroll
                        for (int kk = 0; kk < 4; kk++) {                            // 4 MMAs of 32 bytes of K each per 128-byte row
                            tm_mma<HALF, PAIR>(d, da + kk * step_a, db + kk * step_b, idesc, kk ? 1u : acc);
                            if constexpr (!HALF) tm_mma<HALF, PAIR>(d + 256, da + (A_BYTES >> 4) + kk * step_a, db + kk * step_b, idesc_lo, kk ? 1u : acc);
                        }
                        tm_commit<PAIR>(&empty[s]);
                    }
                    __syncwarp();
                    acc = 1u;
                    if (++s == ST) { s = 0; phase ^= 1u; }
                }
                if (ok && elect_one()) tm_commit<PAIR>(&acc_full[buf]);
                __syncwarp();
            }
        }
    } else {
        // epilogue: warp w owns TMEM lanes 32w .. 32w+31 = rows 32w + lane of the tile
        const uint32_t lane_addr = (uint32_t)(warp * 32) << 16;
        int tl = 0;
        for (int tile = first; tile < p.tiles; tile += step, tl++) {
            const int buf = tl % nbuf, use_b = tl / nbuf;
            bool ok = true;
            if (lane == 0) ok = tm_wait(&acc_full[buf], (uint32_t)use_b & 1u, failed, 64);
            ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
            if (!ok) break;
            tc_fence_after();
            int b, rb, cb;
            tm_locate(p, tile, b, rb, cb);
            const int row = rb * ROWS + row_of_tile + warp * 32 + lane, col0 = cb * BN;
            T *crow = reinterpret_cast<T *>(p.C) + (long long)b * p.c_bs + (long long)row * p.c_rs;
            const bool vec = p.c_cs == 1 && !p.accumulate && ((uintptr_t)crow & 15) == 0;
            const uint32_t d = tmem + lane_addr + (HALF ? buf * 256 : 0);
            float *mine = p.part + ((long long)(tile * p.splits + rank) * TM_BM + warp * 32 + lane) * BN;             // row of the partial tile (splits > 1)
#pragma unroll 1
            for (int c0 = 0; c0 < BN; c0 += 32) {
                uint32_t v[32];
                if constexpr (HALF) { tmem_ld32w(d + c0, v); tmem_wait_ld(); }
                else {
                    // A_hi B_hi and A_hi B_lo: B's parts follow each other (in a pair, for each CTA's half of the columns)
                    uint32_t u[32], x[32];
                    const uint32_t hi = d + c0 + (c0 / BNL) * BNL;
                    tmem_ld32w(hi, v); tmem_ld32w(hi + BNL, u); tmem_ld32w(d + 256 + c0, x);
                    tmem_wait_ld();
#pragma unroll
                    for (int j = 0; j < 32; j++) v[j] = __float_as_uint(__uint_as_float(v[j]) + (__uint_as_float(u[j]) + __uint_as_float(x[j])));
                }
                if (c0 + 32 >= BN) {                                                // the accumulator is in registers: it may be overwritten
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) { if constexpr (PAIR) tm_arrive_at(tm_mapa(smem_u32(&acc_empty[buf]), 0)); else mbar_arrive(&acc_empty[buf]); }
                }
                if (!PAIR && p.splits > 1) {
#pragma unroll
                    for (int j = 0; j < 32; j += 4)
                        *reinterpret_cast<float4 *>(mine + c0 + j) = make_float4(__uint_as_float(v[j]), __uint_as_float(v[j + 1]), __uint_as_float(v[j + 2]), __uint_as_float(v[j + 3]));
                } else if (row < p.N) {
                    // whole groups of 32 columns: straight-line stores, 16 bytes along the row, or element by element where the rows are
                    // the contiguous index (neighbouring lanes then write neighbouring elements)
                    const bool whole = !p.accumulate && col0 + c0 + 32 <= p.M;
                    if (whole && (vec || p.c_rs == 1)) {
                        const T *bias = reinterpret_cast<const T *>(p.bias);
                        const float brow = ld0(p.bias_mode == 1, bias + row);
#pragma unroll
                        for (int j = 0; j < 32; j++) v[j] = __float_as_uint(p.alpha * __uint_as_float(v[j]) + brow);
                        if (p.bias_mode == 2) {
#pragma unroll
                            for (int j = 0; j < 32; j++) v[j] = __float_as_uint(__uint_as_float(v[j]) + ld(bias + col0 + c0 + j));
                        }
                        if (!vec) {
                            T *dst = crow + (long long)(col0 + c0) * p.c_cs;
#pragma unroll
                            for (int j = 0; j < 32; j++, dst += p.c_cs) st(dst, __uint_as_float(v[j]));
                        } else if constexpr (HALF) {
                            uint4 *dst = reinterpret_cast<uint4 *>(crow + col0 + c0);
#pragma unroll
                            for (int j = 0; j < 32; j += 8) {
                                uint32_t w[4];
#pragma unroll
                                for (int q = 0; q < 4; q++) {
                                    const __half2 h = __floats2half2_rn(__uint_as_float(v[j + 2 * q]), __uint_as_float(v[j + 2 * q + 1]));
                                    w[q] = *reinterpret_cast<const uint32_t *>(&h);
                                }
                                dst[j / 8] = make_uint4(w[0], w[1], w[2], w[3]);
                            }
                        } else {
                            uint4 *dst = reinterpret_cast<uint4 *>(crow + col0 + c0);
#pragma unroll
                            for (int j = 0; j < 32; j += 4) dst[j / 4] = make_uint4(v[j], v[j + 1], v[j + 2], v[j + 3]);
                        }
                    } else {
#pragma unroll
                        for (int j = 0; j < 32; j += 4)
                            if (col0 + c0 + j < p.M) {
                                const float r[4] = {__uint_as_float(v[j]), __uint_as_float(v[j + 1]), __uint_as_float(v[j + 2]), __uint_as_float(v[j + 3])};
                                tm_store4<T>(p, crow, row, col0 + c0 + j, r, vec);
                            }
                    }
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (*failed && tid == 0) atomicCAS(p.status, 0, 8);
    if constexpr (PAIR) {
        tm_cluster_sync();                                                          // both CTAs are done with each other's memory
        if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
        tm_cluster_sync();
    } else if (warp == 0) tmem_dealloc(tmem, 512);
}

// C from the partial tiles of a split contraction: a thread per four neighbouring columns; PARTS threads share the partial tiles
// of a quad where there are many (their sums are added in order).
template <class T, int PARTS> __global__ void __launch_bounds__(256) tm_reduce_kernel(const __grid_constant__ TmParams p)
{
    pdl_wait();
    constexpr int Q = 256 / PARTS;                                                  // quads of a block
    __shared__ float4 sums[PARTS > 1 ? PARTS : 1][Q];
    const int quads = p.BN / 4, per = TM_BM * quads, part = threadIdx.x / Q, e = blockIdx.x * Q + threadIdx.x % Q;    // (per is a multiple of 256: a block stays inside one tile)
    const int tile = e / per, in = e - tile * per, r = in / quads, c = (in - r * quads) * 4;
    int b, rb, cb;
    tm_locate(p, tile, b, rb, cb);
    const int row = rb * TM_BM + r, col = cb * p.BN + c;
    const bool live = row < p.N && col < p.M;
    const float4 *src = reinterpret_cast<const float4 *>(p.part + (long long)tile * p.splits * TM_BM * p.BN) + in;
    const int k0 = p.splits * part / PARTS, k1 = p.splits * (part + 1) / PARTS;
    float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
    if (live) {
#pragma unroll 8
        for (int k = k0; k < k1; k++) { const float4 u = src[(long long)k * per]; t.x += u.x; t.y += u.y; t.z += u.z; t.w += u.w; }
    }
    if constexpr (PARTS > 1) {
        sums[part][threadIdx.x % Q] = t;
        __syncthreads();
        if (part > 0) return;
#pragma unroll
        for (int k = 1; k < PARTS; k++) { const float4 u = sums[k][threadIdx.x]; t.x += u.x; t.y += u.y; t.z += u.z; t.w += u.w; }
    }
    if (!live) return;
    T *crow = reinterpret_cast<T *>(p.C) + (long long)b * p.c_bs + (long long)row * p.c_rs;
    const float v[4] = {t.x, t.y, t.z, t.w};
    tm_store4<T>(p, crow, row, col, v, p.c_cs == 1 && !p.accumulate && ((uintptr_t)crow & (4 * sizeof(T) - 1)) == 0);
}

// ---------------------------------------------------------------- operand packing
// dst[(b * rows + r) * Kp + k] = src[b*bs + r*rs + k*cs] for k < K (columns K..Kp-1 are never read: the tensor map ends at K).
// fp32: hi part to dst, lo part to lo.  One launch for both operands of a product.  K-contiguous sources go straight through
// registers, 32 rows x 64 k per block and eight k per thread; the others through a shared-memory tile of 32 k x 64 rows, read
// as vectors along the rows where they are contiguous and aligned, written as whole 128-byte rows of 32 k (64 x [64 x 784]
// transposed and split: 15.5 us with scalar reads of 32 rows, 9.2 us so).
template <class T> struct PackOp { const T *src; T *dst, *lo; long long rs, cs, bs; int rows, K, Kp, nk, nr, first, straight, vec; };
template <class T> struct PackOps { PackOp<T> op[2]; int count; };

template <class T>
__global__ void __launch_bounds__(256) pack_kmajor_kernel(const __grid_constant__ PackOps<T> ops)
{
    pdl_wait();
    __shared__ float tile[32][65];
    const PackOp<T> &o = ops.op[ops.count > 1 && (int)blockIdx.x >= ops.op[1].first ? 1 : 0];
    const int t = (int)blockIdx.x - o.first, tr = t / o.nk, b = tr / o.nr;
    if (!o.straight) {
        const int k0 = (t - tr * o.nk) * 32, r0 = (tr - b * o.nr) * 64, left = o.rows - r0;
        const T *s = o.src + (long long)b * o.bs + (long long)r0 * o.rs;
        if (sizeof(T) == 4 && o.vec) {
            const int rq = (threadIdx.x & 15) * 4, kk = threadIdx.x >> 4;
            float4 v[2];
#pragma unroll
            for (int q = 0; q < 2; q++) {
                const T *p = s + rq + (long long)(k0 + kk + 16 * q) * o.cs;
                v[q] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (k0 + kk + 16 * q < o.K) {
                    if (rq + 4 <= left) v[q] = *reinterpret_cast<const float4 *>(p);
                    else { if (rq < left) v[q].x = ld(p); if (rq + 1 < left) v[q].y = ld(p + 1); if (rq + 2 < left) v[q].z = ld(p + 2); }
                }
            }
#pragma unroll
            for (int q = 0; q < 2; q++) { float *d = &tile[kk + 16 * q][rq]; d[0] = v[q].x; d[1] = v[q].y; d[2] = v[q].z; d[3] = v[q].w; }
        } else {
            const int rr = threadIdx.x & 63, kk = threadIdx.x >> 6;
            const T *p = s + (long long)rr * o.rs + (long long)(k0 + kk) * o.cs;
            float v[8];
#pragma unroll
            for (int q = 0; q < 8; q++, p += 4 * o.cs) v[q] = ld0(rr < left && k0 + kk + 4 * q < o.K, p);
#pragma unroll
            for (int q = 0; q < 8; q++) tile[kk + 4 * q][rr] = v[q];
        }
        __syncthreads();
        const int kq = (threadIdx.x & 7) * 4;
        if (k0 + kq >= o.Kp) return;
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int row = (threadIdx.x >> 3) + 32 * h;
            if (row >= left) return;
            const long long at = ((long long)b * o.rows + r0 + row) * o.Kp + k0 + kq;
            if constexpr (sizeof(T) == 4) {
                uint32_t hi[4], lo[4];
#pragma unroll
                for (int q = 0; q < 4; q++) split_tf32(tile[kq + q][row], hi[q], lo[q]);
                *reinterpret_cast<uint4 *>(o.dst + at) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
                *reinterpret_cast<uint4 *>(o.lo + at) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
            } else {
                const __half2 x = __floats2half2_rn(tile[kq][row], tile[kq + 1][row]), y = __floats2half2_rn(tile[kq + 2][row], tile[kq + 3][row]);
                *reinterpret_cast<uint2 *>(o.dst + at) = make_uint2(*reinterpret_cast<const uint32_t *>(&x), *reinterpret_cast<const uint32_t *>(&y));
            }
        }
        return;
    }
    const int k0 = (t - tr * o.nk) * 64, r0 = (tr - b * o.nr) * 32;
    const T *s = o.src + (long long)b * o.bs;
    const int r = threadIdx.x >> 3, kq = (threadIdx.x & 7) * 8;
    float v[8];
    {
        const T *p = s + (long long)(r0 + r) * o.rs + k0 + kq;
        if (o.vec && r0 + r < o.rows && k0 + kq + 8 <= o.K) {
            if constexpr (sizeof(T) == 4) {
                const float4 x = *reinterpret_cast<const float4 *>(p), y = *reinterpret_cast<const float4 *>(p + 4);
                v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w; v[4] = y.x; v[5] = y.y; v[6] = y.z; v[7] = y.w;
            } else {
#pragma unroll
                for (int q = 0; q < 8; q++) v[q] = ld(p + q);
            }
        } else {
#pragma unroll
            for (int q = 0; q < 8; q++) v[q] = ld0(r0 + r < o.rows && k0 + kq + q < o.K, p + q);
        }
    }
    if (r0 + r >= o.rows || k0 + kq >= o.Kp) return;
    const long long at = ((long long)b * o.rows + r0 + r) * o.Kp + k0 + kq;          // Kp is a multiple of 16 bytes
    if constexpr (sizeof(T) == 4) {
        uint32_t hi[8], lo[8];
#pragma unroll
        for (int q = 0; q < 8; q++) split_tf32(v[q], hi[q], lo[q]);
#pragma unroll
        for (int h = 0; h < 2; h++)
            if (k0 + kq + 4 * h < o.Kp) {
                *reinterpret_cast<uint4 *>(o.dst + at + 4 * h) = make_uint4(hi[4 * h], hi[4 * h + 1], hi[4 * h + 2], hi[4 * h + 3]);
                *reinterpret_cast<uint4 *>(o.lo + at + 4 * h) = make_uint4(lo[4 * h], lo[4 * h + 1], lo[4 * h + 2], lo[4 * h + 3]);
            }
    } else {
        uint32_t w[4];
#pragma unroll
        for (int q = 0; q < 4; q++) { const __half2 h = __floats2half2_rn(v[2 * q], v[2 * q + 1]); w[q] = *reinterpret_cast<const uint32_t *>(&h); }
        *reinterpret_cast<uint4 *>(o.dst + at) = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// inner: extent of the contiguous index, outer: of the other one, `os` elements apart
template <class T> static bool make_map(EncodeTiledFn enc, CUtensorMap *m, const T *base, int inner, int outer, int batch, long long os, long long bs, int box_inner, int box_outer)
{
    cuuint64_t gdim[3] = {(cuuint64_t)inner, (cuuint64_t)outer, (cuuint64_t)batch};
    cuuint64_t gstr[2] = {(cuuint64_t)os * sizeof(T), (cuuint64_t)(batch > 1 ? bs : (long long)outer * os) * sizeof(T)};
    cuuint32_t box[3] = {(cuuint32_t)box_inner, (cuuint32_t)box_outer, 1u};
    cuuint32_t estr[3] = {1, 1, 1};
    return enc(m, sizeof(T) == 2 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, (void *)base, gdim, gstr, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Tile and CTAs per tile with the fewest cycles by a model of the main loop, fitted to measured products: a K step costs its
// tensor time or what its bytes take from L2 into an SM (58 bytes per cycle with every SM loading, 81 with half of them); a CTA
// pair's K step a third more than its tensor time; a tile 2500 cycles beside its K steps; a launch 2000, of pairs 10000; the
// pass over the partial tiles of a split contraction a launch and their bytes.  So pairs take the products of several rounds of
// tiles with long contractions (fp16 4096^3: 97 us against 105 us) and single CTAs the rest (fp16 2048^3: 17.6 us against
// 19.1 us, fp32 1000 x 600 x 1300: 16.2 us against 19.5 us).
template <class T> static void tm_plan(int N, int M, int batch, int ksteps, int most_splits, int &BN, int &splits, int &pair)
{
    constexpr bool HALF = sizeof(T) == 2;
    double best = 1e30;
    const int bns_h[4] = {256, 128, 64, 256}, bns_f[4] = {128, 96, 64, 128};
    for (int i = 0; i < 4; i++) {
        const bool two = i == 3;
        const int bn = HALF ? bns_h[i] : bns_f[i], rows = two ? 2 * TM_BM : TM_BM;
        const long long tiles = (long long)ceil_div(N, rows) * ceil_div(M, bn) * batch;
        for (int s = 1; s <= (two ? 1 : most_splits); s++) {
            if (s > 1 && (ksteps < 2 * s || tiles * s > sm_count())) break;
            const long long ctas = tiles * s * (two ? 2 : 1);
            const double tensor = (HALF ? 2.0 : 6.0) * bn * (two ? 4.0 / 3.0 : 1.0);
            const double fill = (HALF ? 1 : 2) * 128.0 * (128 + (two ? bn / 2 : bn)) / (ctas <= sm_count() / 2 ? 81.0 : 58.0);
            const double reduce = s > 1 ? 4000.0 + 512.0 * bn * tiles * s / 2000.0 : 0.0;
            const double cost = (two ? 10000.0 : 2000.0) + (double)ceil_div(ctas, sm_count()) * (std::max(tensor, fill) * ceil_div(ksteps, s) + 2500.0) + reduce;
            if (cost < 0.97 * best) { best = cost; BN = bn; splits = s; pair = two ? 1 : 0; }
        }
    }
}

// fp16 operands stay where they are when one index is contiguous (returns 1: the contracted one, 2: the rows) and the other steps in
// multiples of 16 bytes; 0 = the operand is packed
template <class T> static int tm_in_place(const T *src, long long rs, long long cs, long long bs, int rows, int K, int batch)
{
    constexpr long long EB = 16 / (long long)sizeof(T);
    if (sizeof(T) != 2 || ((uintptr_t)src & 15) || (batch > 1 && bs % EB)) return 0;
    return cs == 1 && rs % EB == 0 && rs >= K ? 1 : rs == 1 && cs % EB == 0 && cs >= rows ? 2 : 0;
}

// false: no tensor-map encoder, no memory for the copies
template <class T> static bool tm_product(const GemmDesc<T> &d)
{
    typedef TmCfg<T> Cfg;
    EncodeTiledFn enc = (EncodeTiledFn)tc_encode_tiled_fn();
    int *status = tc_status_word();
    if (!enc || !status) return false;
    Scope sc;
    if (!sc.ok()) return false;
    constexpr long long EB = 16 / (long long)sizeof(T);
    const int Kp = (int)(((long long)d.K + EB - 1) / EB * EB);
    struct Op { const T *hi, *lo; long long os, bs; int mn; };
    PackOps<T> pack;
    pack.count = 0;
    int blocks = 0;
    auto prepare = [&](const T *src, long long rs, long long cs, long long bs, int rows, int batch, Op &o) -> bool {
        const int where = tm_in_place<T>(src, rs, cs, bs, rows, d.K, batch);
        if (where) { o = {src, nullptr, where == 1 ? rs : cs, bs, where - 1}; return true; }
        const size_t count = ((size_t)batch * rows * Kp + 63) & ~(size_t)63;
        T *hi = sc.try_scratch<T>(Cfg::PARTS * count), *lo = sizeof(T) == 4 ? hi + count : nullptr;
        if (!hi) return false;
        PackOp<T> &q = pack.op[pack.count++];
        const bool straight = cs == 1;
        q = {src, hi, lo, rs, cs, bs, rows, d.K, Kp, ceil_div(Kp, straight ? 64 : 32), ceil_div(rows, straight ? 32 : 64), blocks, straight, (straight ? rs : rs == 1 ? cs : 1) % EB == 0 && (batch == 1 || bs % EB == 0) && ((uintptr_t)src & 15) == 0};
        blocks += q.nk * q.nr * batch;
        o = {hi, lo, Kp, (long long)rows * Kp, 0};
        return true;
    };
    Op a, b;
    const int copies = d.batch * d.segs, b_batch = d.segs == 1 && d.b_bs == 0 ? 1 : copies;      // a batch and the segments of a contraction are walked alike
    if (!prepare(d.A, d.a_rs, d.a_cs, d.segs > 1 ? d.a_ks : d.a_bs, d.N, copies, a)) return false;
    if (!prepare(d.B, d.b_cs, d.b_rs, d.segs > 1 ? d.b_ks : d.b_bs, d.M, b_batch, b)) return false;     // row of the B operand = column of C
    TmParams p;
    p.kps = ceil_div(d.K, Cfg::BK); p.ksteps = p.kps * d.segs;
    p.BN = sizeof(T) == 2 ? 256 : 128; p.splits = 1; p.pair = 0;
    tm_plan<T>(d.N, d.M, d.batch, p.ksteps, d.segs > 1 ? 1 << 20 : 8, p.BN, p.splits, p.pair);
    p.C = d.C; p.bias = d.bias; p.N = d.N; p.M = d.M; p.K = d.K;
    p.c_rs = d.c_rs; p.c_cs = d.c_cs; p.c_bs = d.c_bs;
    p.alpha = d.alpha; p.accumulate = d.accumulate ? 1 : 0; p.bias_mode = d.bias ? d.bias_mode : 0;
    p.status = status; p.a_mn = a.mn; p.b_mn = b.mn; p.b_one = b_batch < copies;
    p.tiles_m = ceil_div(d.M, p.BN); p.tiles_n = ceil_div(d.N, p.pair ? 2 * TM_BM : TM_BM); p.tiles = p.tiles_m * p.tiles_n * d.batch;
    p.part = nullptr;
    if (p.splits > 1 && !(p.part = sc.try_scratch<float>((size_t)p.tiles * p.splits * TM_BM * p.BN))) return false;
    const int b_rows = p.pair ? p.BN / 2 : p.BN;
    p.stage_bytes = Cfg::PARTS * (TM_BM * 128u + (uint32_t)b_rows * 128u);
    p.stages = std::min<int>(TM_MAX_STAGES, TM_RING / p.stage_bytes);
    auto map = [&](CUtensorMap *m, const T *base, const Op &o, int rows, int batch, int box_rows) {
        return o.mn ? make_map<T>(enc, m, base, rows, d.K, batch, o.os, o.bs, 64, 64) : make_map<T>(enc, m, base, d.K, rows, batch, o.os, o.bs, Cfg::BK, box_rows);
    };
    CUtensorMap ma0, ma1, mb0, mb1;
    if (!map(&ma0, a.hi, a, d.N, copies, TM_BM) || !map(&mb0, b.hi, b, d.M, b_batch, b_rows)) return false;
    ma1 = ma0; mb1 = mb0;
    if (sizeof(T) == 4 && (!map(&ma1, a.lo, a, d.N, copies, TM_BM) || !map(&mb1, b.lo, b, d.M, b_batch, b_rows))) return false;
    if (pack.count) TL_LAUNCH((pack_kmajor_kernel<T>), blocks, 256, 0, pack);
    const size_t smem = (size_t)p.stages * p.stage_bytes + 1024;
    static bool attr_set = false;
    if (!attr_set) {
        cudaFuncSetAttribute(gemm_tma_kernel<T, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(TM_RING + 1024));
        cudaFuncSetAttribute(gemm_tma_kernel<T, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(TM_RING + 1024));
        attr_set = true;
    }
    if (p.pair) TL_LAUNCH_CLUSTER((gemm_tma_kernel<T, true>), (unsigned)(2 * std::min(p.tiles, sm_count() / 2)), TM_THREADS, smem, 2, ma0, ma1, mb0, mb1, p);
    else if (p.splits == 1) TL_LAUNCH((gemm_tma_kernel<T, false>), (unsigned)std::min(p.tiles, sm_count()), TM_THREADS, smem, ma0, ma1, mb0, mb1, p);
    else TL_LAUNCH((gemm_tma_kernel<T, false>), (unsigned)(p.tiles * p.splits), TM_THREADS, smem, ma0, ma1, mb0, mb1, p);
    profile_add_flops(d.flops);
    if (p.splits > 1) {
        const long long quads = (long long)p.tiles * TM_BM * p.BN / 4;
        if (p.splits <= 16) TL_LAUNCH((tm_reduce_kernel<T, 1>), (unsigned)(quads / 256), 256, 0, p);
        else TL_LAUNCH((tm_reduce_kernel<T, 8>), (unsigned)(quads / 32), 256, 0, p);
    }
    return true;
}

// The packed copies of a batch are scratch that the library keeps (in fp32 twice the bytes of the operand), so a batch that would need
// more than this goes out in slices (a block of 512 MB then holds those of the shared operand too); a slice's launches are hundreds of
// microseconds by then.
static constexpr long long TM_PACK_BYTES = 480ll << 20;

// Returns false when the product should go to the other kernels (too small, or see tm_product).
template <class T> bool gemm_tensor_core_tma(const GemmDesc<T> &d)
{
    typedef TmCfg<T> Cfg;
    if (d.N < 1 || d.M < 1 || d.K < 1 || d.batch < 1 || d.segs < 1 || (d.batch > 1 && d.segs > 1)) return false;
    if (gemm_path() != 3) {      // 3 = forced (tests): every shape, the tails come from the tensor maps' zero fill
        if (d.segs == 1 && (d.N < TM_BM || d.M < TM_BM / 2 || d.K < (d.batch > 1 ? 1 : 2) * Cfg::BK)) return false;
        if ((long long)d.N * d.M * d.K * d.batch * d.segs < (1ll << 26)) return false;
    }
    if (d.batch == 1 || d.accumulate) return tm_product<T>(d);           // (accumulated: a slice that fails could not be taken back)
    const long long bytes = (long long)sizeof(T) * Cfg::PARTS * d.K;
    const long long per = (tm_in_place<T>(d.A, d.a_rs, d.a_cs, d.a_bs, d.N, d.K, d.batch) ? 0 : bytes * d.N) +
                          (d.b_bs == 0 || tm_in_place<T>(d.B, d.b_cs, d.b_rs, d.b_bs, d.M, d.K, d.batch) ? 0 : bytes * d.M);
    const int slices = ceil_div(d.batch, per ? std::max(1ll, TM_PACK_BYTES / per) : d.batch), each = ceil_div(d.batch, slices);
    for (int b = 0; b < d.batch; b += each) {
        GemmDesc<T> s = d;
        s.batch = std::min(each, d.batch - b);
        s.A += b * d.a_bs; s.B += b * d.b_bs; s.C += b * d.c_bs;
        s.flops = d.flops * s.batch / d.batch;
        if (!tm_product<T>(s)) return false;
    }
    return true;
}
template bool gemm_tensor_core_tma<float>(const GemmDesc<float> &);
template bool gemm_tensor_core_tma<__half>(const GemmDesc<__half> &);

} // namespace tl

// Output projection of the attention layer on the 5th-generation tensor cores:
//   out[b, s, n] = sum_{h, d} attn[b, h, s, d] * W[n, h * D + d]  (+ bias[n])
// i.e. the reference's  attn_output.transpose(1, 2).reshape([b, q_len, hidden]) -> Linear::forward
// (models/kalosm-llama/src/raw/attention_layer.rs:450-454, fusor-ml/fusor/src/layers/linear.rs:72-115) with a dense bf16
// weight.  The transpose is never materialised: the A operand tile [128 rows of s][64 of d] of head h is exactly one TMA
// box of the [B, Hq, S, D] attention output, so a K step of the GEMM is "head h, half of d".
//
// Four kernels, picked by how many output tiles there are (launch_out_proj):
//   oproj_pair_kernel   many tiles: a CTA pair (cta_group::2) owns 256 x 256 outputs,
//   oproj_single_kernel one CTA per 128 x 256 outputs, where that fills the waves better,
//   oproj_split_kernel  fewer 128 x 128 tiles than SMs: a cluster of up to 8 CTAs shares a tile along K,
//   oproj_rows_kernel   a few rows (decode): the weight streams through warp MMAs, no tile of A at all.
#pragma once
#include <cuda.h>

#include "ptx_sm100.cuh"

namespace fusor {

constexpr int OP_BM = 128, OP_BK = 64;
constexpr int OP_A_BYTES = OP_BM * OP_BK * 2;
constexpr int OP_THREADS = 192;  // warp 0 producer, warp 1 TMEM + MMA, warps 2-5 epilogue

struct OprojParams {
    int B, Hq, S, D, N;
    int m_tiles_per_batch, n_tiles, k_chunks;  // K = Hq * D in chunks of 64
    int n_group;                               // n tiles per raster group (their weight rows stay in L2 while all m sweep by)
    const float* bias;                         // [N] or null
    int out_dtype;                             // 0 f32, 1 bf16
    int* err;
    // plain pointers for the kernels that do not go through tensor maps
    const __nv_bfloat16* a;
    long long as[3];                           // element strides of batch, head and row
    const __nv_bfloat16* w;
    long long ws;                              // element stride of a weight row
    void* out;
    long long os[2];                           // element strides of batch and row
};

// ------------------------------------------------------------------------------------------------- CTA pairs, 256 x 256
// Bound: tensor pipe.  One CTA with a 128 x 256 tile fetches 48 KB per 512 tensor cycles = 96 B/clk, twice what L2 delivers
// to all SMs at once (46 B/clk/SM), and reads 12 KB of shared memory per 128 cycles.  A pair shares the weight tile: each
// CTA holds its own 128 rows of A and half of the 256 weight rows, 32 KB per 512 cycles and 8 KB per 128, which also makes
// room for six stages.  The two row tiles of a pair are neighbours in (batch, row) order and need not be of one batch.
// Persistent pairs, two 256-column accumulators: the epilogue of a tile (TMEM -> registers -> + bias -> swizzled staging ->
// TMA store) runs under the main loop of the next.  The leader (CTA 0) issues every MMA; loads of both CTAs signal its
// barriers, its commits signal both.  All waits are bounded.
// 16384 rows, K = N = 4096: 448 us with single CTAs of 128 x 256, 411 us as pairs (1338 TFLOP/s); 4096 rows, K = N = 8192:
// 422 and 364 us (1512 TFLOP/s).
constexpr int OP2_BN = 256, OP2_STAGES = 6;
constexpr int OP2_B_BYTES = (OP2_BN / 2) * OP_BK * 2;
constexpr int OP2_STAGE_BYTES = OP_A_BYTES + OP2_B_BYTES;
constexpr int OP2_OUT_STAGE = 32 * 128;  // per epilogue warp and buffer: 32 rows x 128 bytes
constexpr size_t OP2_SMEM_BYTES = 1024 + (size_t)OP2_STAGES * OP2_STAGE_BYTES + 4 * 2 * (size_t)OP2_OUT_STAGE + 256;

// Tile order: groups of n_group neighbouring n tiles; inside a group every pair of row tiles in turn, n fastest.  The
// group's weight rows (n_group x 256 x K x 2 bytes, sized by the host to about a quarter of L2) stay resident while the A
// panels stream by; with a weight that fits L2 whole there is one group and A is read once.
__device__ __forceinline__ void op_tile_coords(const OprojParams& P, int m_total, int tile, int& nt, int& mt) {
    const int g = tile / (P.n_group * m_total);
    const int r = tile - g * P.n_group * m_total;
    const int width = min(P.n_group, P.n_tiles - g * P.n_group);
    mt = r / width;
    nt = g * P.n_group + r % width;
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(OP_THREADS, 1)
    oproj_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmW,
                      const __grid_constant__ CUtensorMap tmO, const OprojParams P) {
    extern __shared__ uint8_t op_smem_raw[];
    uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(op_smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* ring = base;                                  // [stage]{A 16 KB, half of B 16 KB}
    uint8_t* out_sm = ring + OP2_STAGES * OP2_STAGE_BYTES;  // [4 warps][2 buffers] x 4 KB
    uint64_t* bars = reinterpret_cast<uint64_t*>(out_sm + 4 * 2 * OP2_OUT_STAGE);
    uint64_t* full = bars;                             // [6] the leader's: loads of both CTAs
    uint64_t* empty = bars + OP2_STAGES;               // [6] both CTAs', by the leader's commits
    uint64_t* acc_full = bars + 2 * OP2_STAGES;        // [2] both CTAs', by the leader's commits
    uint64_t* acc_empty = bars + 2 * OP2_STAGES + 2;   // [2] the leader's: the 8 epilogue warps of the pair
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * OP2_STAGES + 4);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t rank = cluster_cta_rank();
    const int n_pairs = (int)gridDim.x / 2, pair = (int)blockIdx.x / 2;
    const int m_tiles = P.B * P.m_tiles_per_batch, m_pairs = (m_tiles + 1) / 2;
    const int n_tiles_total = m_pairs * P.n_tiles;
    const int d_chunks = P.D / OP_BK;  // K chunks per head

    if (tid == 0) {
        for (int i = 0; i < OP2_STAGES; ++i) {
            mbar_init(full + i, 1);
            mbar_init(empty + i, 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(acc_full + i, 1);
            mbar_init(acc_empty + i, 8);
        }
        *abort_flag = 0;
        mbar_fence_init();
        tma_prefetch_desc(&tmA);
        tma_prefetch_desc(&tmW);
        tma_prefetch_desc(&tmO);
    }
    if (warp == 1) {
        tmem_alloc_pair(tmem_slot, 512);
        tmem_relinquish_pair();
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();  // the other CTA's barriers are initialised before anything signals them
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer (both CTAs)
        if (elect_one_sync()) {
            int it = 0;  // K steps loaded so far
            bool ok = true;
            for (int tile = pair; tile < n_tiles_total && ok; tile += n_pairs) {
                int nt, mp;
                op_tile_coords(P, m_pairs, tile, nt, mp);
                // an odd number of row tiles: the last pair's second CTA repeats its neighbour's rows and stores nothing
                const int mt = min(2 * mp + (int)rank, m_tiles - 1);
                const int b = mt / P.m_tiles_per_batch, s0 = (mt % P.m_tiles_per_batch) * OP_BM;
                for (int kc = 0; kc < P.k_chunks; ++kc, ++it) {
                    const int st = it % OP2_STAGES, use = it / OP2_STAGES;
                    if (use > 0 && !mbar_wait_cluster(empty + st, (use - 1) & 1, abort_flag, P.err, 60)) { ok = false; break; }
                    uint8_t* a_sm = ring + st * OP2_STAGE_BYTES;
                    if (rank == 0) mbar_arrive_expect_tx(full + st, 2 * OP2_STAGE_BYTES);
                    const uint32_t bar = map_to_cta(full + st, 0);
                    tma_load_4d_pair(a_sm, &tmA, bar, (kc % d_chunks) * OP_BK, s0, kc / d_chunks, b);
                    tma_load_4d_pair(a_sm + OP_A_BYTES, &tmW, bar, kc * OP_BK, nt * OP2_BN + (int)rank * (OP2_BN / 2), 0, 0);
                }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer (leader only)
        if (rank == 0 && elect_one_sync()) {
            constexpr uint32_t idesc = make_idesc_f16(1, 1, 0, 0, 2 * OP_BM, OP2_BN);
            const uint64_t a_desc0 = make_smem_desc_sw128(smem_u32(ring), 16, 1024);
            const uint64_t b_desc0 = make_smem_desc_sw128(smem_u32(ring + OP_A_BYTES), 16, 1024);
            int it = 0, tc = 0;  // K steps consumed, tiles started
            bool ok = true;
            for (int tile = pair; tile < n_tiles_total && ok; tile += n_pairs, ++tc) {
                const int ab = tc & 1;
                // the accumulator is free once the epilogues of the tile before last have read it out
                if (tc >= 2 && !mbar_wait_cluster(acc_empty + ab, ((tc >> 1) - 1) & 1, abort_flag, P.err, 61)) break;
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + ab * OP2_BN;
                for (int kc = 0; kc < P.k_chunks; ++kc, ++it) {
                    const int st = it % OP2_STAGES;
                    if (!mbar_wait_cluster(full + st, (it / OP2_STAGES) & 1, abort_flag, P.err, 62)) { ok = false; break; }
                    tc_fence_after();
                    const uint64_t off = (uint64_t)((st * OP2_STAGE_BYTES) >> 4);
#pragma unroll
                    for (int kk = 0; kk < OP_BK / 16; ++kk)
                        tc_mma_ss_pair(d_tmem, a_desc0 + off + (uint64_t)((kk * 32) >> 4), b_desc0 + off + (uint64_t)((kk * 32) >> 4),
                                       idesc, (kc > 0 || kk > 0));
                    tc_commit_pair(empty + st);
                }
                if (ok) tc_commit_pair(acc_full + ab);
            }
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------------------ epilogue (both CTAs, each its own rows)
        const int quad = warp & 3;  // TMEM lane quadrant of this warp
        const uint32_t lane_base = (uint32_t)(quad * 32) << 16;
        uint8_t* stage0 = out_sm + (warp - 2) * 2 * OP2_OUT_STAGE;
        int tc = 0, stores = 0;
        bool ok = true;
        for (int tile = pair; tile < n_tiles_total && ok; tile += n_pairs, ++tc) {
            int nt, mp;
            op_tile_coords(P, m_pairs, tile, nt, mp);
            const int mt = 2 * mp + (int)rank;
            const int b = mt / P.m_tiles_per_batch, s0 = (mt % P.m_tiles_per_batch) * OP_BM;
            const int ab = tc & 1;
            const int row_g = s0 + quad * 32;
            const bool mine = mt < m_tiles && row_g < P.S;
            ok = __all_sync(0xffffffffu, mbar_wait_cluster(acc_full + ab, (tc >> 1) & 1, abort_flag, P.err, 63));
            if (!ok) break;
            tc_fence_after();
            const uint32_t acc = tmem_base + lane_base + ab * OP2_BN;
#pragma unroll 1
            for (int cc = 0; cc < OP2_BN / 32; ++cc) {
                float v[32];
                tmem_ld32(acc + cc * 32, *reinterpret_cast<uint32_t(*)[32]>(&v[0]));
                tc_wait_ld();
                if (cc == OP2_BN / 32 - 1) {
                    // the accumulator has been read out: the leader may start the tile after next in it
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_cluster(map_to_cta(acc_empty + ab, 0));
                }
                if (P.bias != nullptr) {
                    // every lane reads the same 32 values (one broadcast per load); columns past N are never stored
                    const int n0 = nt * OP2_BN + cc * 32;
#pragma unroll
                    for (int i = 0; i < 32; ++i) v[i] += (n0 + i < P.N) ? __ldg(P.bias + n0 + i) : 0.0f;
                }
                uint8_t* stage = stage0 + (stores & 1) * OP2_OUT_STAGE;
                uint8_t* my = stage + lane * 128;
                if (P.out_dtype == 0) {
                    if (stores >= 2) {
                        if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
                        __syncwarp();
                    }
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        *reinterpret_cast<float4*>(my + ((i ^ (lane & 7)) << 4)) = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
                    fence_proxy_async_smem();
                    __syncwarp();
                    if (lane == 0) {
                        if (mine && nt * OP2_BN + cc * 32 < P.N) tma_store_4d(&tmO, stage, nt * OP2_BN + cc * 32, row_g, 0, b);
                        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                    }
                    ++stores;
                } else {
                    // bf16: two chunks of 32 columns fill one 128-byte row
                    if ((cc & 1) == 0 && stores >= 2) {
                        if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
                        __syncwarp();
                    }
                    const int ch0 = (cc & 1) * 4;
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        *reinterpret_cast<uint4*>(my + (((ch0 + i) ^ (lane & 7)) << 4)) =
                            make_uint4(pack_bf16(v[8 * i], v[8 * i + 1]), pack_bf16(v[8 * i + 2], v[8 * i + 3]),
                                       pack_bf16(v[8 * i + 4], v[8 * i + 5]), pack_bf16(v[8 * i + 6], v[8 * i + 7]));
                    if (cc & 1) {
                        fence_proxy_async_smem();
                        __syncwarp();
                        if (lane == 0) {
                            if (mine && nt * OP2_BN + (cc - 1) * 32 < P.N) tma_store_4d(&tmO, stage, nt * OP2_BN + (cc - 1) * 32, row_g, 0, b);
                            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                        }
                        ++stores;
                    }
                }
            }
        }
        if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        __syncwarp();
    }
    // ---- teardown: every role falls through to here, also after a timeout.  Neither CTA leaves while the other may still
    // signal its barriers.
    tc_fence_before();
    __syncthreads();
    cluster_sync();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc_pair(tmem_base, 512);
    }
}

// ------------------------------------------------------------------------------------------- single CTAs, 128 x 256
// The same pipeline with one CTA per tile, 4-stage ring (48 KB per stage), warp 0 producer, warp 1 MMA, warps 2-5 epilogue.  Half
// the tile of a pair, so it stays where whole waves of pairs would be left nearly empty (4700 rows, K = N = 1024: 76 pair tiles
// on 74 pairs take 18.0 us, 148 single ones 12.1), and in a single wave of few K steps, where the pair's cluster barriers
// show (2000 rows, K 1024, N 2048: 13.4 and 13.0 us; K 1536 15.2 and 15.0; K 2048 18.3 and 18.7).
constexpr int OP1_BN = 256, OP1_STAGES = 4;
constexpr int OP1_STAGE_BYTES = OP_A_BYTES + OP1_BN * OP_BK * 2;
constexpr size_t OP1_SMEM_BYTES = 1024 + (size_t)OP1_STAGES * OP1_STAGE_BYTES + 4 * 2 * (size_t)OP2_OUT_STAGE + 256;

__global__ void __launch_bounds__(OP_THREADS, 1)
    oproj_single_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmW,
                       const __grid_constant__ CUtensorMap tmO, const OprojParams P) {
    extern __shared__ uint8_t op_smem_raw[];
    uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(op_smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* ring = base;                                      // [stage]{A 16 KB, B 32 KB}
    uint8_t* out_sm = ring + OP1_STAGES * OP1_STAGE_BYTES;        // [4 warps][2 buffers] x 4 KB
    uint64_t* bars = reinterpret_cast<uint64_t*>(out_sm + 4 * 2 * OP2_OUT_STAGE);
    uint64_t* full = bars;                   // [4]
    uint64_t* empty = bars + OP1_STAGES;      // [4]
    uint64_t* acc_full = bars + 2 * OP1_STAGES;       // [2]
    uint64_t* acc_empty = bars + 2 * OP1_STAGES + 2;  // [2]
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * OP1_STAGES + 4);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n_tiles_total = P.B * P.m_tiles_per_batch * P.n_tiles;
    const int d_chunks = P.D / OP_BK;  // K chunks per head

    if (tid == 0) {
        for (int i = 0; i < OP1_STAGES; ++i) {
            mbar_init(full + i, 1);
            mbar_init(empty + i, 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(acc_full + i, 1);
            mbar_init(acc_empty + i, 4);
        }
        *abort_flag = 0;
        mbar_fence_init();
        tma_prefetch_desc(&tmA);
        tma_prefetch_desc(&tmW);
        tma_prefetch_desc(&tmO);
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer
        if (elect_one_sync()) {
            int it = 0;  // K steps loaded so far: ring slot it % 4
            bool ok = true;
            for (int tile = blockIdx.x; tile < n_tiles_total && ok; tile += gridDim.x) {
                int nt, mt;
                op_tile_coords(P, P.B * P.m_tiles_per_batch, tile, nt, mt);
                const int b = mt / P.m_tiles_per_batch, s0 = (mt % P.m_tiles_per_batch) * OP_BM;
                for (int kc = 0; kc < P.k_chunks; ++kc, ++it) {
                    const int st = it % OP1_STAGES, use = it / OP1_STAGES;
                    if (use > 0 && !mbar_wait(empty + st, (use - 1) & 1, abort_flag, P.err, 60)) { ok = false; break; }
                    uint8_t* a_sm = ring + st * OP1_STAGE_BYTES;
                    mbar_arrive_expect_tx(full + st, OP1_STAGE_BYTES);
                    tma_load_4d(a_sm, &tmA, full + st, (kc % d_chunks) * OP_BK, s0, kc / d_chunks, b);
                    tma_load_4d(a_sm + OP_A_BYTES, &tmW, full + st, kc * OP_BK, nt * OP1_BN, 0, 0);
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer
        if (elect_one_sync()) {
            constexpr uint32_t idesc = make_idesc_f16(1, 1, 0, 0, OP_BM, OP1_BN);
            const uint64_t a_desc0 = make_smem_desc_sw128(smem_u32(ring), 16, 1024);
            const uint64_t b_desc0 = make_smem_desc_sw128(smem_u32(ring + OP_A_BYTES), 16, 1024);
            int it = 0, tc = 0;  // K steps consumed, tiles started
            bool ok = true;
            for (int tile = blockIdx.x; tile < n_tiles_total && ok; tile += gridDim.x, ++tc) {
                const int ab = tc & 1;
                // the accumulator is free once the epilogue of the tile before last has read it out
                if (tc >= 2 && !mbar_wait(acc_empty + ab, ((tc >> 1) - 1) & 1, abort_flag, P.err, 61)) break;
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + ab * OP1_BN;
                for (int kc = 0; kc < P.k_chunks; ++kc, ++it) {
                    const int st = it % OP1_STAGES;
                    if (!mbar_wait(full + st, (it / OP1_STAGES) & 1, abort_flag, P.err, 62)) { ok = false; break; }
                    tc_fence_after();
                    const uint64_t off = (uint64_t)((st * OP1_STAGE_BYTES) >> 4);
#pragma unroll
                    for (int kk = 0; kk < OP_BK / 16; ++kk)
                        tc_mma_ss(d_tmem, a_desc0 + off + (uint64_t)((kk * 32) >> 4), b_desc0 + off + (uint64_t)((kk * 32) >> 4),
                                  idesc, (kc > 0 || kk > 0));
                    tc_commit(empty + st);
                }
                if (ok) tc_commit(acc_full + ab);
            }
        }
    } else {
        // ------------------------------------------------------------------ epilogue
        const int quad = warp & 3;  // TMEM lane quadrant of this warp
        const uint32_t lane_base = (uint32_t)(quad * 32) << 16;
        uint8_t* stage0 = out_sm + (warp - 2) * 2 * OP2_OUT_STAGE;
        int tc = 0, stores = 0;
        bool ok = true;
        for (int tile = blockIdx.x; tile < n_tiles_total && ok; tile += gridDim.x, ++tc) {
            int nt, mt;
            op_tile_coords(P, P.B * P.m_tiles_per_batch, tile, nt, mt);
            const int b = mt / P.m_tiles_per_batch, s0 = (mt % P.m_tiles_per_batch) * OP_BM;
            const int ab = tc & 1;
            const int row_g = s0 + quad * 32;
            ok = mbar_wait(acc_full + ab, (tc >> 1) & 1, abort_flag, P.err, 63);
            if (!ok) break;
            tc_fence_after();
            const uint32_t acc = tmem_base + lane_base + ab * OP1_BN;
#pragma unroll 1
            for (int cc = 0; cc < OP1_BN / 32; ++cc) {
                float v[32];
                tmem_ld32(acc + cc * 32, *reinterpret_cast<uint32_t(*)[32]>(&v[0]));
                tc_wait_ld();
                if (cc == OP1_BN / 32 - 1) {
                    // the accumulator has been read out: the MMA warp may start the tile after next in it
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(acc_empty + ab);
                }
                if (P.bias != nullptr) {
                    // every lane reads the same 32 values (one broadcast per load); columns past N are never stored
                    const int n0 = nt * OP1_BN + cc * 32;
#pragma unroll
                    for (int i = 0; i < 32; ++i) v[i] += (n0 + i < P.N) ? __ldg(P.bias + n0 + i) : 0.0f;
                }
                if (P.out_dtype == 0) {
                    uint8_t* stage = stage0 + (stores & 1) * OP2_OUT_STAGE;
                    if (stores >= 2) {
                        if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
                        __syncwarp();
                    }
                    uint8_t* my = stage + lane * 128;
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        *reinterpret_cast<float4*>(my + ((i ^ (lane & 7)) << 4)) = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
                    fence_proxy_async_smem();
                    __syncwarp();
                    if (lane == 0) {
                        if (row_g < P.S && nt * OP1_BN + cc * 32 < P.N) tma_store_4d(&tmO, stage, nt * OP1_BN + cc * 32, row_g, 0, b);
                        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                    }
                    ++stores;
                } else {
                    // bf16: two chunks of 32 columns fill one 128-byte row
                    uint8_t* stage = stage0 + (stores & 1) * OP2_OUT_STAGE;
                    if ((cc & 1) == 0 && stores >= 2) {
                        if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
                        __syncwarp();
                    }
                    uint8_t* my = stage + lane * 128;
                    const int ch0 = (cc & 1) * 4;
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        *reinterpret_cast<uint4*>(my + (((ch0 + i) ^ (lane & 7)) << 4)) =
                            make_uint4(pack_bf16(v[8 * i], v[8 * i + 1]), pack_bf16(v[8 * i + 2], v[8 * i + 3]),
                                       pack_bf16(v[8 * i + 4], v[8 * i + 5]), pack_bf16(v[8 * i + 6], v[8 * i + 7]));
                    if (cc & 1) {
                        fence_proxy_async_smem();
                        __syncwarp();
                        if (lane == 0) {
                            if (row_g < P.S && nt * OP1_BN + (cc - 1) * 32 < P.N)
                                tma_store_4d(&tmO, stage, nt * OP1_BN + (cc - 1) * 32, row_g, 0, b);
                            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                        }
                        ++stores;
                    }
                }
            }
        }
        if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
    }
    // ---- teardown: every role falls through to here, also after a timeout
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
}

// ------------------------------------------------------------------------------------------- 128 x 128 tiles, K split
// Fewer tiles than SMs: bound by how fast the SMs that have work pull weights, so a cluster of KS CTAs takes one tile, each
// a KS-th of K.  The partial sums meet in shared memory: CTA r owns 128 / KS columns of the tile, the others store theirs
// into its slots (float4 per row and 4 columns, so that neighbouring lanes write neighbouring addresses), and it adds them
// up in rank order: the result does not depend on timing.  Against 128 x 256 tiles without a split, K = N = 4096: 128 rows
// 31.0 -> 14.6 us, 400 rows 29.5 -> 25.2 us; K = N = 1024, 128 rows: 11.6 -> 7.7 us.
constexpr int OPS_BN = 128, OPS_STAGES = 4, OPS_MAX_SPLIT = 8;
constexpr int OPS_B_BYTES = OPS_BN * OP_BK * 2;
constexpr int OPS_STAGE_BYTES = OP_A_BYTES + OPS_B_BYTES;
constexpr int OPS_RED_BYTES = OP_BM * OPS_BN * 4;  // KS slots of 128 x (128 / KS) f32, the own one unused
constexpr size_t OPS_SMEM_BYTES = 1024 + (size_t)OPS_STAGES * OPS_STAGE_BYTES + OPS_RED_BYTES + 256;

__global__ void __launch_bounds__(OP_THREADS, 1)
    oproj_split_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmW, const OprojParams P, const int ks) {
    extern __shared__ uint8_t op_smem_raw[];
    uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(op_smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* ring = base;
    uint8_t* red = ring + OPS_STAGES * OPS_STAGE_BYTES;  // [source rank][column group of 4][row] float4
    uint64_t* bars = reinterpret_cast<uint64_t*>(red + OPS_RED_BYTES);
    uint64_t* full = bars;                 // [4]
    uint64_t* empty = bars + OPS_STAGES;   // [4]
    uint64_t* acc_full = bars + 2 * OPS_STAGES;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * OPS_STAGES + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rank = (int)cluster_cta_rank();  // part of K (the cluster is ks CTAs along x)
    const int tile = (int)blockIdx.x / ks;
    const int mt = tile / P.n_tiles, nt = tile % P.n_tiles;
    const int b = mt / P.m_tiles_per_batch, s0 = (mt % P.m_tiles_per_batch) * OP_BM;
    const int k_begin = (int)((long long)P.k_chunks * rank / ks), k_end = (int)((long long)P.k_chunks * (rank + 1) / ks);
    const int d_chunks = P.D / OP_BK;

    if (tid == 0) {
        for (int i = 0; i < OPS_STAGES; ++i) {
            mbar_init(full + i, 1);
            mbar_init(empty + i, 1);
        }
        mbar_init(acc_full, 1);
        *abort_flag = 0;
        mbar_fence_init();
        tma_prefetch_desc(&tmA);
        tma_prefetch_desc(&tmW);
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, OPS_BN);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    bool ok = true;
    if (warp == 0) {
        if (elect_one_sync()) {
            for (int kc = k_begin; kc < k_end; ++kc) {
                const int it = kc - k_begin, st = it % OPS_STAGES, use = it / OPS_STAGES;
                if (use > 0 && !mbar_wait(empty + st, (use - 1) & 1, abort_flag, P.err, 64)) break;
                uint8_t* a_sm = ring + st * OPS_STAGE_BYTES;
                mbar_arrive_expect_tx(full + st, OPS_STAGE_BYTES);
                tma_load_4d(a_sm + OP_A_BYTES, &tmW, full + st, kc * OP_BK, nt * OPS_BN, 0, 0);
                tma_load_4d(a_sm, &tmA, full + st, (kc % d_chunks) * OP_BK, s0, kc / d_chunks, b);
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        if (elect_one_sync()) {
            constexpr uint32_t idesc = make_idesc_f16(1, 1, 0, 0, OP_BM, OPS_BN);
            const uint64_t a_desc0 = make_smem_desc_sw128(smem_u32(ring), 16, 1024);
            const uint64_t b_desc0 = make_smem_desc_sw128(smem_u32(ring + OP_A_BYTES), 16, 1024);
            bool good = true;
            for (int kc = k_begin; kc < k_end; ++kc) {
                const int it = kc - k_begin, st = it % OPS_STAGES;
                if (!mbar_wait(full + st, (it / OPS_STAGES) & 1, abort_flag, P.err, 65)) { good = false; break; }
                tc_fence_after();
                const uint64_t off = (uint64_t)((st * OPS_STAGE_BYTES) >> 4);
#pragma unroll
                for (int kk = 0; kk < OP_BK / 16; ++kk)
                    tc_mma_ss(tmem_base, a_desc0 + off + (uint64_t)((kk * 32) >> 4), b_desc0 + off + (uint64_t)((kk * 32) >> 4), idesc,
                              (it > 0 || kk > 0));
                tc_commit(empty + st);
            }
            if (good) tc_commit(acc_full);
        }
        __syncwarp();
    }
    const int quad = warp & 3, row = quad * 32 + lane;
    const uint32_t acc = tmem_base + ((uint32_t)(quad * 32) << 16);
    const int width = OPS_BN / ks;  // columns a CTA of the cluster finishes: 128, 64, 32 or 16
    if (warp >= 2) {
        ok = __all_sync(0xffffffffu, mbar_wait(acc_full, 0, abort_flag, P.err, 66));
        tc_fence_after();
    }
    if (ks > 1) {
        cluster_sync();  // every CTA of the cluster has started: its shared memory may be written
        if (warp >= 2 && ok) {
            for (int c16 = 0; c16 < OPS_BN / 16; ++c16) {
                const int owner = c16 * 16 / width;
                if (owner == rank) continue;
                float v[16];
                tmem_ld16(acc + c16 * 16, *reinterpret_cast<uint32_t(*)[16]>(&v[0]));
                tc_wait_ld();
                const int g0 = (c16 * 16 - owner * width) / 4;
                const uint32_t dst = map_to_cta(red, (uint32_t)owner) + (uint32_t)((((rank * width / 4) + g0) * OP_BM + row) * 16);
#pragma unroll
                for (int i = 0; i < 4; ++i) st_cluster_f4(dst + i * OP_BM * 16, make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]));
            }
        }
        __syncwarp();
        cluster_sync();  // all partial sums have arrived, and none is still on its way to a CTA that leaves
    }
    if (warp >= 2 && ok) {
        const bool row_ok = s0 + row < P.S;
        const long long o_row = (long long)b * P.os[0] + (long long)(s0 + row) * P.os[1];
        for (int c16 = 0; c16 < width / 16; ++c16) {
            float v[16];
            const int c0 = rank * width + c16 * 16;
            tmem_ld16(acc + c0, *reinterpret_cast<uint32_t(*)[16]>(&v[0]));
            tc_wait_ld();
            if (ks > 1) {
                float sum[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) sum[i] = 0.0f;
                for (int r = 0; r < ks; ++r) {
                    if (r == rank) {
#pragma unroll
                        for (int i = 0; i < 16; ++i) sum[i] += v[i];
                    } else {
                        const float4* src = reinterpret_cast<const float4*>(red) + ((r * width / 4) + c16 * 4) * OP_BM + row;
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const float4 f = src[i * OP_BM];
                            sum[4 * i] += f.x; sum[4 * i + 1] += f.y; sum[4 * i + 2] += f.z; sum[4 * i + 3] += f.w;
                        }
                    }
                }
#pragma unroll
                for (int i = 0; i < 16; ++i) v[i] = sum[i];
            }
            const int n0 = nt * OPS_BN + c0;
            if (P.bias != nullptr) {
#pragma unroll
                for (int i = 0; i < 16; ++i) v[i] += (n0 + i < P.N) ? __ldg(P.bias + n0 + i) : 0.0f;
            }
            if (!row_ok) {
                // nothing to store
            } else if (n0 + 16 <= P.N) {
                if (P.out_dtype == 0) {
                    float4* o = reinterpret_cast<float4*>(reinterpret_cast<float*>(P.out) + o_row + n0);
#pragma unroll
                    for (int i = 0; i < 4; ++i) o[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
                } else {
                    uint4* o = reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(P.out) + o_row + n0);
#pragma unroll
                    for (int i = 0; i < 2; ++i)
                        o[i] = make_uint4(pack_bf16(v[8 * i], v[8 * i + 1]), pack_bf16(v[8 * i + 2], v[8 * i + 3]),
                                          pack_bf16(v[8 * i + 4], v[8 * i + 5]), pack_bf16(v[8 * i + 6], v[8 * i + 7]));
                }
            } else {
#pragma unroll
                for (int i = 0; i < 16; ++i)
                    if (n0 + i < P.N) st_from_float(P.out, P.out_dtype, o_row + n0 + i, v[i]);
            }
            __syncwarp();  // the next tcgen05.ld takes the whole warp
        }
    }
    // ---- teardown: every role falls through to here, also after a timeout
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, OPS_BN);
    }
}

// ----------------------------------------------------------------------------------------------------- a few rows
// Decode: HBM-bound on the weight, read once.  A CTA owns 16 weight rows (the 16-row operand of m16n8k16) and its warps take
// 64-wide chunks of K in turn; the activations are the 8-column operand.  Both operands come straight from global memory,
// 16 bytes per lane: a lane's 8 consecutive k stand for the fragment's (2t, 2t+1, 2t+8, 2t+9) of two MMAs, the same
// permutation of k on both sides.  The warps' sums meet in shared memory and are added in warp order.
// K = N = 4096, up to 16 rows: 30.5 us on 128 x 256 tiles, 10.4 us here (3.2 TB/s); K = N = 8192: 57 and 29 to 32 us; the
// split kernel takes 14.2 us at 17 rows, so the line is where the two-group operand ends.
constexpr int OPR_WARPS = 8, OPR_MAX_ROWS = 16;

template <int NT>  // 8-row groups of activations: rows <= 8 NT
__global__ void __launch_bounds__(OPR_WARPS * 32) oproj_rows_kernel(const OprojParams P) {
    __shared__ float part[OPR_WARPS][16][8 * NT + 1];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, kq = (lane & 3) * 8;
    const int n0 = blockIdx.x * 16, rows = P.B * P.S;
    const __nv_bfloat16* w0 = P.w + (long long)min(n0 + g, P.N - 1) * P.ws + kq;
    const __nv_bfloat16* w1 = P.w + (long long)min(n0 + g + 8, P.N - 1) * P.ws + kq;
    const __nv_bfloat16* x[NT];
    bool live[NT];
#pragma unroll
    for (int j = 0; j < NT; ++j) {
        const int r = j * 8 + g;
        live[j] = r < rows;
        const int rr = live[j] ? r : 0;
        x[j] = P.a + (long long)(rr / P.S) * P.as[0] + (long long)(rr % P.S) * P.as[2] + kq;
    }
    float c[NT][4];
#pragma unroll
    for (int j = 0; j < NT; ++j) c[j][0] = c[j][1] = c[j][2] = c[j][3] = 0.0f;
    const int d_chunks = P.D / OP_BK;
    constexpr int U = 4;  // chunks in flight per warp: 8 KB of weights
    for (int kc0 = warp; kc0 < P.k_chunks; kc0 += OPR_WARPS * U) {
        uint4 wa[U][4];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int kc = kc0 + u * OPR_WARPS;
            if (kc < P.k_chunks) {
                wa[u][0] = __ldcs(reinterpret_cast<const uint4*>(w0 + (long long)kc * OP_BK));
                wa[u][1] = __ldcs(reinterpret_cast<const uint4*>(w1 + (long long)kc * OP_BK));
                wa[u][2] = __ldcs(reinterpret_cast<const uint4*>(w0 + (long long)kc * OP_BK + 32));
                wa[u][3] = __ldcs(reinterpret_cast<const uint4*>(w1 + (long long)kc * OP_BK + 32));
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int kc = kc0 + u * OPR_WARPS;
            if (kc < P.k_chunks) {
                const long long a_off = (long long)(kc / d_chunks) * P.as[1] + (kc % d_chunks) * OP_BK;
#pragma unroll
                for (int j = 0; j < NT; ++j) {
                    uint4 xa = make_uint4(0, 0, 0, 0), xb = xa;
                    if (live[j]) {
                        xa = __ldg(reinterpret_cast<const uint4*>(x[j] + a_off));
                        xb = __ldg(reinterpret_cast<const uint4*>(x[j] + a_off + 32));
                    }
                    const uint32_t f0[4] = {wa[u][0].x, wa[u][1].x, wa[u][0].y, wa[u][1].y};
                    const uint32_t f1[4] = {wa[u][0].z, wa[u][1].z, wa[u][0].w, wa[u][1].w};
                    const uint32_t f2[4] = {wa[u][2].x, wa[u][3].x, wa[u][2].y, wa[u][3].y};
                    const uint32_t f3[4] = {wa[u][2].z, wa[u][3].z, wa[u][2].w, wa[u][3].w};
                    mma_bf16_16816(c[j], f0, xa.x, xa.y);
                    mma_bf16_16816(c[j], f1, xa.z, xa.w);
                    mma_bf16_16816(c[j], f2, xb.x, xb.y);
                    mma_bf16_16816(c[j], f3, xb.z, xb.w);
                }
            }
        }
    }
    const int cq = (lane & 3) * 2;
#pragma unroll
    for (int j = 0; j < NT; ++j) {
        part[warp][g][j * 8 + cq] = c[j][0];
        part[warp][g][j * 8 + cq + 1] = c[j][1];
        part[warp][g + 8][j * 8 + cq] = c[j][2];
        part[warp][g + 8][j * 8 + cq + 1] = c[j][3];
    }
    __syncthreads();
    for (int i = tid; i < 16 * rows; i += OPR_WARPS * 32) {
        const int n = n0 + (i & 15), r = i >> 4;
        if (n >= P.N) continue;
        float v = 0.0f;
#pragma unroll
        for (int w = 0; w < OPR_WARPS; ++w) v += part[w][i & 15][r];
        if (P.bias != nullptr) v += __ldg(P.bias + n);
        st_from_float(P.out, P.out_dtype, (long long)(r / P.S) * P.os[0] + (long long)(r % P.S) * P.os[1] + n, v);
    }
}

}  // namespace fusor

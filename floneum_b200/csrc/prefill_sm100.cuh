// Causal / full flash-attention prefill on the 5th-generation tensor cores (tcgen05 + TMEM).
//
// One CTA owns a 128-row query tile of one (batch, query head) and walks the PF_BN-key tiles it can see
// (causal tile skip).  Two CTAs are resident per SM (256 TMEM columns and <= 113 KB of shared memory each),
// so the softmax of one overlaps the tensor work, prologue and epilogue of the other.  Roles, by warp:
//   warp 0      TMA producer: Q once, then K and V tiles into PF_SBUF-slot rings (128-byte swizzle, CTA-local loads).
//   warp 1      allocates TMEM and issues every tcgen05.mma from one thread:
//               S_j = Q K_j^T   (SS: both operands in shared memory, K-major, N = PF_BN),
//               O  += P_j V_j   (TS: P read from TMEM, V from shared memory, MN-major, N = 128),
//               and the next S into the buffer P_j is read from straight after (the pipe runs in issue order).
//   warps 2-5   softmax: a thread per query row reads S from TMEM, keeps the running max / sum, writes P
//               (16-bit) back over S, rescales O in TMEM only when the row max has grown by more than 2^8
//               (lazy rescale), and finally writes O / l.
// TMEM columns: S / P buffers from column 0 (PF_SBUF x PF_BN <= 128), O in [128,256).
// All waits are bounded (ptx_sm100.cuh); on a timeout the CTA unwinds and frees its TMEM.
//
// SPLIT: a chain of tiles takes about a microsecond each whatever else runs, so a call with few query tiles (a follow-up on
// a warm cache, few heads) leaves most SMs idle for the length of its longest row of tiles.  A cluster of up to 8 CTAs then
// shares the key tiles of one query tile.  Each part ends with its own (m, l, O); the parts swap (m, l) through shared
// memory over the cluster, scale their O to the common maximum and sum, and push the columns another CTA finishes into its
// (idle) Q / K / V buffers; every CTA adds its 128 / C columns up in rank order and stores them.
// H32/8, 64 new rows on 4000 cached keys 53 -> 24 us, 200 on 1000 20.0 -> 18.3 us; H8/1, 300 on 3000 44 -> 21 us; H8/8 S2048
// causal 30 -> 23 us.  The merge costs 4 to 6 us, so 12 tiles are not split (14.8 us, 16.8 in two parts).
//
// Replaces the reference's fused kernel for Sq > 1
// (fusor-ml/core/src/composite/flash_attention.rs:147-331: one subgroup per output row,
// keys visited serially, mask read from a dense [Sq,Skv] tensor).
#pragma once
#include <cuda.h>

#include "ptx_sm100.cuh"

namespace fusor {

#ifndef PF_BN_CFG
#define PF_BN_CFG 64
#endif
#ifndef PF_SBUF_CFG
#define PF_SBUF_CFG 2
#endif
constexpr int PF_BM = 128, PF_BN = PF_BN_CFG, PF_D = 128;
constexpr int PF_SBUF = PF_SBUF_CFG;           // S buffers in TMEM = K / V ring slots
constexpr int PF_THREADS = 64 + 128;           // warp 0 TMA, warp 1 MMA, then softmax warps (warp % 4 = TMEM lane quadrant), a thread per query row
constexpr int PF_Q_BYTES = PF_BM * PF_D * 2;   // two [128][64] halves
constexpr int PF_Q_HALF = PF_Q_BYTES / 2;
constexpr int PF_KV_BYTES = PF_BN * PF_D * 2;  // two [PF_BN][64] halves
constexpr int PF_KV_HALF = PF_KV_BYTES / 2;
constexpr uint32_t PF_TMEM_COLS = 256;
constexpr uint32_t PF_COL_S = 0, PF_COL_O = 128;  // S buffer b at PF_COL_S + PF_BN b
constexpr float PF_RESCALE_THRESHOLD = 8.0f;      // in log2 units
static_assert(PF_SBUF * PF_BN <= 128 && PF_BN % 32 == 0, "tile configuration");

struct PrefillParams {
    void* out;
    int out_dtype;             // 0 f32, 1 bf16, 2 f16
    long long os[3];           // element strides of batch, head, row
    int B, Hq, Hkv, Sq, Skv;
    int causal;
    int window;                // > 0: sliding window on top of causal (key k allowed iff q + off - window < k <= q + off)
    float scale_log2;
    int n_q_tiles;
    int* err;
    const int* v_f16_overflow; // written by the V pre-pass: non-zero when some |v| does not fit f16; null = no f16 copy
    int in_f16;                // q, k and v are f16 (else bf16): f16 weights against V itself, no copy, no fallback
    const float* kmask;        // optional additive key mask [B][Skv] f32 (MaskKind::BatchKeyMask), added to the scaled scores
    long long kmask_stride;    // elements between batches
    float kmask_mul;           // 1 / scale: the mask is added to the raw scores as mask / scale, before the common scaling
    const float* qkmask;       // optional additive mask [Sq][Skv] f32 (MaskKind::QKMask), shared by batches and heads; 64-key kernel only
    long long qkmask_stride;   // elements between query rows
};

constexpr int PF_MAX_SPLIT = 8;
constexpr size_t PF_SMEM_BYTES = 1024 + (size_t)PF_Q_BYTES + 2 * PF_SBUF * (size_t)PF_KV_BYTES + 512 + 2 * PF_MAX_SPLIT * 128 * 4;
static_assert(PF_Q_BYTES + 2 * PF_SBUF * PF_KV_BYTES >= PF_BM * PF_D * 4, "the parts' columns fit the operand buffers");

// Two raw scores += mask / scale.  Finite values down to the lowest float would overflow to -inf in the quotient, and a row in which
// every key carries them would be NaN instead of the mean of V: they are held at a floor, next to which a score disappears as it
// does next to the value itself.  -inf stays -inf by the product with the least float, which is below 5e-7 for any other value.
// For the same reason the maximum of a row stays in raw units where there is a mask tensor, and differences are taken before the
// scaling: s scale - max of such values would not be 0 where s is the maximum.
__device__ __forceinline__ void prefill_mask(const PrefillParams& P, float m0, float m1, float& s0, float& s1) {
    const float2 m = make_float2(m0, m1), x = fmul2(m, make_float2(P.kmask_mul, P.kmask_mul));
    const float2 s = fadd2(ffma2(m, make_float2(0x1p-149f, 0x1p-149f), make_float2(s0, s1)), make_float2(fmaxf(x.x, -1e38f), fmaxf(x.y, -1e38f)));
    s0 = s.x;
    s1 = s.y;
}

// s += the mask values `row` holds for the N keys from k0 on, four at a time where they are aligned and all there
template <int N>
__device__ __forceinline__ void prefill_add_mask(const PrefillParams& P, const float* row, int k0, float (&s)[N]) {
    const float* m = row + k0;
    if (k0 + N <= P.Skv && reinterpret_cast<uintptr_t>(m) % 16 == 0) {
#pragma unroll
        for (int i = 0; i < N; i += 4) {
            const float4 x = __ldg(reinterpret_cast<const float4*>(m + i));
            prefill_mask(P, x.x, x.y, s[i], s[i + 1]);
            prefill_mask(P, x.z, x.w, s[i + 2], s[i + 3]);
        }
    } else {
#pragma unroll
        for (int i = 0; i < N; i += 2) prefill_mask(P, __ldg(row + min(k0 + i, P.Skv - 1)), __ldg(row + min(k0 + i + 1, P.Skv - 1)), s[i], s[i + 1]);
    }
}

// s -= m
template <int N>
__device__ __forceinline__ void prefill_subtract(float m, float (&s)[N]) {
#pragma unroll
    for (int i = 0; i < N; i += 2) {
        const float2 x = fadd2(make_float2(s[i], s[i + 1]), make_float2(-m, -m));
        s[i] = x.x;
        s[i + 1] = x.y;
    }
}

// P (the softmax weights handed to the second MMA) and V must have the same 16-bit type: kind::f16 rejects a
// mixed f16 / bf16 operand pair.  bf16 weights (8 significant bits) put rows with few keys above the 2e-3
// tolerance, so the host converts V to f16 once per call (cast_v_to_f16_kernel) and the kernel keeps P in f16
// (11 bits).  When some |v| exceeds the f16 range the pre-pass raises a flag and every CTA falls back to bf16
// P with the original bf16 V: the choice is a uniform runtime branch (descriptor bits and the tensor map).
// MASK: 0 = no mask tensor, 1 = a key mask, 2 = an [Sq, Skv] mask
template <bool SPLIT, int MASK>
__global__ void __launch_bounds__(PF_THREADS, 2)
    prefill_sm100_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                         const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmV16,
                         const __grid_constant__ CUtensorMap tmO, const PrefillParams P, const int parts) {
    extern __shared__ uint8_t pf_smem_raw[];
    uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(pf_smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* q_sm = base;
    uint8_t* k_sm = q_sm + PF_Q_BYTES;             // PF_SBUF slots
    uint8_t* v_sm = k_sm + PF_SBUF * PF_KV_BYTES;  // PF_SBUF slots
    uint64_t* bars = reinterpret_cast<uint64_t*>(v_sm + PF_SBUF * PF_KV_BYTES);
    uint64_t* q_full = bars + 0;
    uint64_t* k_full = bars + 1;    // [2]
    uint64_t* k_empty = bars + 3;   // [2]
    uint64_t* v_full = bars + 5;    // [2]
    uint64_t* v_empty = bars + 7;   // [2]
    uint64_t* s_full = bars + 9;    // [2]
    uint64_t* p_full = bars + 11;   // [2]
    uint64_t* pv_done = bars + 13;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 18);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    float2* part_ml = reinterpret_cast<float2*>(bars + 32);  // SPLIT: [part][128 rows] (m, l)

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool use_f16 = P.in_f16 != 0 || (P.v_f16_overflow != nullptr && *P.v_f16_overflow == 0);

    // ---- which tile: heavy (late) query tiles first; consecutive CTAs share a kv head
    const int heads_total = P.Hq * P.B;
    const int part = SPLIT ? (int)cluster_cta_rank() : 0, tile = SPLIT ? (int)blockIdx.x / parts : (int)blockIdx.x;
    const int qt = P.n_q_tiles - 1 - tile / heads_total;
    const int hb = tile % heads_total;
    const int h = hb % P.Hq, b = hb / P.Hq;
    const int hk = h / (P.Hq / P.Hkv);
    const int q0 = qt * PF_BM;
    const int offset = P.Skv - P.Sq;
    int n_kv = (P.Skv + PF_BN - 1) / PF_BN;  // becomes the number of key tiles this CTA visits, starting at tile j_begin
    if (P.causal) n_kv = min(n_kv, (q0 + PF_BM - 1 + offset) / PF_BN + 1);
    int j_begin = P.window > 0 ? max(0, q0 + offset - P.window + 1) / PF_BN : 0;
    n_kv -= j_begin;
    if (SPLIT) {  // this part's tiles; none if there are fewer tiles than parts
        const int first = n_kv * part / parts, last = n_kv * (part + 1) / parts;
        j_begin += first;
        n_kv = last - first;
    }

    if (tid == 0) {
        mbar_init(q_full, 1);
        for (int i = 0; i < 2; ++i) {
            mbar_init(k_full + i, 1);
            mbar_init(k_empty + i, 1);
            mbar_init(v_full + i, 1);
            mbar_init(v_empty + i, 1);
            mbar_init(s_full + i, 1);
            mbar_init(p_full + i, 128);
        }
        mbar_init(pv_done, 1);
        *abort_flag = 0;
        mbar_fence_init();
        tma_prefetch_desc(&tmQ);
        tma_prefetch_desc(&tmK);
        tma_prefetch_desc(use_f16 ? &tmV16 : &tmV);
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, PF_TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    float m_ref = -INFINITY, l = 0.0f;  // of this thread's row (softmax warps)
    const float m_unit = MASK ? P.scale_log2 : 1.0f;  // m_ref times this is in log2 units
    bool ok = true;

    if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer
        if (elect_one_sync()) {
            const CUtensorMap* tv = use_f16 ? &tmV16 : &tmV;
            mbar_arrive_expect_tx(q_full, PF_Q_BYTES);
            tma_load_4d(q_sm, &tmQ, q_full, 0, q0, h, b);
            tma_load_4d(q_sm + PF_Q_HALF, &tmQ, q_full, 64, q0, h, b);
            for (int j = 0; j < n_kv; ++j) {
                const int st = j % PF_SBUF, use = j / PF_SBUF;
                if (use > 0 && !mbar_wait(k_empty + st, (use - 1) & 1, abort_flag, P.err)) break;
                mbar_arrive_expect_tx(k_full + st, PF_KV_BYTES);
                tma_load_4d(k_sm + st * PF_KV_BYTES, &tmK, k_full + st, 0, (j_begin + j) * PF_BN, hk, b);
                tma_load_4d(k_sm + st * PF_KV_BYTES + PF_KV_HALF, &tmK, k_full + st, 64, (j_begin + j) * PF_BN, hk, b);
                if (use > 0 && !mbar_wait(v_empty + st, (use - 1) & 1, abort_flag, P.err)) break;
                mbar_arrive_expect_tx(v_full + st, PF_KV_BYTES);
                tma_load_4d(v_sm + st * PF_KV_BYTES, tv, v_full + st, 0, (j_begin + j) * PF_BN, hk, b);
                tma_load_4d(v_sm + st * PF_KV_BYTES + PF_KV_HALF, tv, v_full + st, 64, (j_begin + j) * PF_BN, hk, b);
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer
        if (elect_one_sync()) {
            // S = Q K^T : A, B bf16, both K-major, M = 128, N = PF_BN
            const uint32_t idesc_qk = P.in_f16 ? make_idesc_f16(0, 0, 0, 0, PF_BM, PF_BN) : make_idesc_f16(1, 1, 0, 0, PF_BM, PF_BN);
            // O += P V  : A = P (TMEM, K-major), B = V MN-major, M = 128, N = D; both f16 or both bf16
            const uint32_t idesc_pv = use_f16 ? make_idesc_f16(0, 0, 0, 1, PF_BM, PF_D) : make_idesc_f16(1, 1, 0, 1, PF_BM, PF_D);
            // descriptors are built once; a k-step or a ring slot only moves the start-address field (units of 16 bytes)
            const uint64_t q_desc0 = make_smem_desc_sw128(smem_u32(q_sm), 16, 1024);
            const uint64_t k_desc0 = make_smem_desc_sw128(smem_u32(k_sm), 16, 1024);
            const uint64_t v_desc0 = make_smem_desc_sw128(smem_u32(v_sm), PF_KV_HALF, 1024);
            auto issue_qk = [&](int j) {  // K tile j (ring slot j % PF_SBUF) -> S buffer j % PF_SBUF
                const int st = j % PF_SBUF;
                const uint64_t k_desc = k_desc0 + (uint64_t)((st * PF_KV_BYTES) >> 4);
                const uint32_t d_tmem = tmem_base + PF_COL_S + st * PF_BN;
#pragma unroll
                for (int kk = 0; kk < PF_D / 16; ++kk) {
                    tc_mma_ss(d_tmem, q_desc0 + (uint64_t)(((kk >> 2) * PF_Q_HALF + (kk & 3) * 32) >> 4),
                              k_desc + (uint64_t)(((kk >> 2) * PF_KV_HALF + (kk & 3) * 32) >> 4), idesc_qk, kk > 0);
                }
                tc_commit(s_full + st);
                tc_commit(k_empty + st);
            };
            ok = mbar_wait(q_full, 0, abort_flag, P.err);
            for (int t = 0; t < PF_SBUF && t < n_kv && ok; ++t) {
                ok = mbar_wait(k_full + t, 0, abort_flag, P.err);
                if (ok) {
                    tc_fence_after();
                    issue_qk(t);
                }
            }
            for (int j = 0; j < n_kv && ok; ++j) {
                const int st = j % PF_SBUF, ph = (j / PF_SBUF) & 1;
                ok = mbar_wait(p_full + st, ph, abort_flag, P.err) && mbar_wait(v_full + st, ph, abort_flag, P.err);
                if (!ok) break;
                tc_fence_after();
                const uint64_t v_desc = v_desc0 + (uint64_t)((st * PF_KV_BYTES) >> 4);
#pragma unroll
                for (int kk = 0; kk < PF_BN / 16; ++kk) {
                    // 16 keys per step: 8 TMEM columns of packed P, 16 rows (2 KB) of the V tile
                    tc_mma_ts(tmem_base + PF_COL_O, tmem_base + PF_COL_S + st * PF_BN + kk * 8,
                              v_desc + (uint64_t)((kk * 2048) >> 4), idesc_pv, (j > 0 || kk > 0));
                }
                tc_commit(v_empty + st);
                tc_commit(pv_done);
                if (j + PF_SBUF < n_kv) {
                    // the next S for this buffer overwrites the columns P_j is being read from: issue order = execution order
                    ok = mbar_wait(k_full + st, ((j + PF_SBUF) / PF_SBUF) & 1, abort_flag, P.err);
                    if (!ok) break;
                    tc_fence_after();
                    issue_qk(j + PF_SBUF);
                }
            }
        }
    } else {
        // ------------------------------------------------------------------ softmax / correction / epilogue
        const int quad = warp & 3;
        const int row = quad * 32 + lane;                        // 0..127 = TMEM lane = query row of the tile
        const uint32_t lane_base = (uint32_t)(quad * 32) << 16;  // this warp's TMEM lane quadrant
        const int qi = q0 + row;
        const int k_limit = P.causal ? min(P.Skv - 1, qi + offset) : P.Skv - 1;  // last key this row may see
        const int k_first = P.window > 0 ? qi + offset - P.window + 1 : 0;      // first key this row may see
        const float c = P.scale_log2;
        const float thr = MASK ? PF_RESCALE_THRESHOLD / c : PF_RESCALE_THRESHOLD;
        const uint32_t o_tmem = tmem_base + lane_base + PF_COL_O;
        for (int j = 0; j < n_kv && ok; ++j) {
            const int st = j % PF_SBUF;
            const uint32_t s_tmem = tmem_base + lane_base + PF_COL_S + st * PF_BN;
            ok = mbar_wait(s_full + st, (j / PF_SBUF) & 1, abort_flag, P.err);
            if (!ok) break;
            tc_fence_after();
            float s[PF_BN];
#pragma unroll
            for (int cc = 0; cc < PF_BN / 32; ++cc)
                tmem_ld32(s_tmem + cc * 32, *reinterpret_cast<uint32_t(*)[32]>(&s[cc * 32]));
            tc_wait_ld();
            const int k0 = (j_begin + j) * PF_BN;
            if (MASK == 1) {
                // additive key mask of this batch row: (s + mask / scale) * scale = s * scale + mask; every thread of the
                // CTA reads the same values (broadcast loads); keys past Skv are cut by the edge mask below
                const float* mk = P.kmask + (long long)b * P.kmask_stride;
                prefill_add_mask(P, mk, k0, s);
            }
            if (MASK == 2) {
                // additive [Sq, Skv] mask tensor: each thread reads its own row's values for this tile (-inf entries give
                // -inf scores, which the code below treats like keys outside a window); no tile can be skipped
                const float* mr = P.qkmask + (long long)min(qi, P.Sq - 1) * P.qkmask_stride;
                prefill_add_mask(P, mr, k0, s);
            }
            if (k0 + PF_BN - 1 > k_limit || k0 < k_first) {  // diagonal, ragged or window-edge tile: mask in the raw domain
#pragma unroll
                for (int i = 0; i < PF_BN; ++i)
                    if (k0 + i > k_limit || k0 + i < k_first) s[i] = -INFINITY;
            }
            float mx[8];
#pragma unroll
            for (int a = 0; a < 8; ++a) mx[a] = fmaxf(s[4 * a], s[4 * a + 1]);
#pragma unroll
            for (int a = 0; a < 8; ++a) mx[a] = fmax3(mx[a], s[4 * a + 2], s[4 * a + 3]);
#pragma unroll
            for (int i = 32; i < PF_BN; i += 16)
#pragma unroll
                for (int a = 0; a < 8; ++a) mx[a] = fmax3(mx[a], s[i + 2 * a], s[i + 2 * a + 1]);
            float pmax = fmaxf(fmax3(mx[0], mx[1], mx[2]), fmaxf(fmax3(mx[3], mx[4], mx[5]), fmaxf(mx[6], mx[7])));
            const float tmax = MASK ? pmax : pmax * c;  // scale > 0
            // lazy rescale: keep the reference max until the true max has moved by more than the threshold
            const float m_new = (tmax > m_ref + thr) ? tmax : m_ref;  // also taken on the first tile
            // A row whose keys so far are all outside its window keeps m = -inf: its weights are exp2(-inf - 0) = 0
            // and its O row stays 0, without a NaN from (-inf) - (-inf).
            const float alpha = (m_new == -INFINITY) ? 1.0f : fast_exp2((m_ref - m_new) * m_unit);  // 1 when unchanged, 0 on a row's first tile
            m_ref = m_new;
            float m_sub = (m_ref == -INFINITY) ? 0.0f : m_ref;
            if (MASK) {
                prefill_subtract(m_sub, s);
                m_sub = 0.0f;
            }
            const float2 c2 = make_float2(c, c), nm2 = make_float2(-m_sub, -m_sub);
            float2 ps0 = make_float2(0.0f, 0.0f), ps1 = make_float2(0.0f, 0.0f);
#pragma unroll
            for (int cc = 0; cc < PF_BN / 32; ++cc) {
                uint32_t pk[16];
#pragma unroll
                for (int i = 0; i < 16; i += 2) {
                    const float2 t0 = ffma2(make_float2(s[cc * 32 + 2 * i], s[cc * 32 + 2 * i + 1]), c2, nm2);
                    const float2 t1 = ffma2(make_float2(s[cc * 32 + 2 * i + 2], s[cc * 32 + 2 * i + 3]), c2, nm2);
                    const float2 p0 = make_float2(fast_exp2(t0.x), fast_exp2(t0.y));
                    const float2 p1 = make_float2(fast_exp2(t1.x), fast_exp2(t1.y));
                    ps0 = fadd2(ps0, p0);
                    ps1 = fadd2(ps1, p1);
                    pk[i] = use_f16 ? pack_f16(p0.x, p0.y) : pack_bf16(p0.x, p0.y);
                    pk[i + 1] = use_f16 ? pack_f16(p1.x, p1.y) : pack_bf16(p1.x, p1.y);
                }
                tmem_st16(s_tmem + cc * 16, pk);  // P overwrites the first PF_BN/2 columns of this S buffer
            }
            l = l * alpha + ((ps0.x + ps0.y) + (ps1.x + ps1.y));
            tc_wait_st();
            if (j > 0) {
                // O must be complete up to tile j-1 before it is rescaled and before P_j is handed over
                ok = mbar_wait(pv_done, (j - 1) & 1, abort_flag, P.err);
                if (!ok) break;
                tc_fence_after();
                if (__any_sync(0xffffffffu, alpha != 1.0f)) {
                    const float2 a2 = make_float2(alpha, alpha);
#pragma unroll
                    for (int cc = 0; cc < 128 / 32; ++cc) {
                        float orr[32];
                        tmem_ld32(o_tmem + cc * 32, *reinterpret_cast<uint32_t(*)[32]>(&orr[0]));
                        tc_wait_ld();
#pragma unroll
                        for (int i = 0; i < 32; i += 2) {
                            const float2 r = fmul2(make_float2(orr[i], orr[i + 1]), a2);
                            orr[i] = r.x;
                            orr[i + 1] = r.y;
                        }
                        tmem_st32(o_tmem + cc * 32, *reinterpret_cast<uint32_t(*)[32]>(&orr[0]));
                    }
                    tc_wait_st();
                }
            }
            tc_fence_before();
            mbar_arrive(p_full + st);
        }
        if (ok && (!SPLIT || n_kv > 0)) ok = mbar_wait(pv_done, (n_kv - 1) & 1, abort_flag, P.err);
        // Epilogue: O / l goes through shared memory (the Q / K / V buffers are idle once the last MMA has
        // completed) in the 128-byte-swizzled layout of the output tensor map, then out with TMA stores:
        // full 128-byte lines instead of one 16-byte piece per row per instruction.  Rows past Sq are clipped.
        constexpr int BLK_BYTES = 128 * 128;  // one [128 rows][128 bytes] column block
        if (!SPLIT && ok) {
            tc_fence_after();
            const float inv_l = 1.0f / l;
#pragma unroll
            for (int cc = 0; cc < 128 / 32; ++cc) {
                float orr[32];
                tmem_ld32(o_tmem + cc * 32, *reinterpret_cast<uint32_t(*)[32]>(&orr[0]));
                tc_wait_ld();
                const int col0 = cc * 32;  // first output column of this chunk
                if (P.out_dtype == 0) {
                    // f32: 32 columns = one 128-byte block row = 8 chunks of 16 bytes
                    uint8_t* blk = base + (col0 / 32) * BLK_BYTES + row * 128;
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        *reinterpret_cast<float4*>(blk + ((i ^ (row & 7)) << 4)) =
                            make_float4(orr[4 * i] * inv_l, orr[4 * i + 1] * inv_l, orr[4 * i + 2] * inv_l, orr[4 * i + 3] * inv_l);
                } else {
                    // bf16 / f16: 32 columns = half of a 128-byte block row = 4 chunks of 16 bytes
                    uint8_t* blk = base + (col0 / 64) * BLK_BYTES + row * 128;
                    const int ch0 = (col0 % 64) / 8;
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        *reinterpret_cast<uint4*>(blk + (((ch0 + i) ^ (row & 7)) << 4)) =
                            make_uint4(pack_16(P.out_dtype, orr[8 * i] * inv_l, orr[8 * i + 1] * inv_l),
                                       pack_16(P.out_dtype, orr[8 * i + 2] * inv_l, orr[8 * i + 3] * inv_l),
                                       pack_16(P.out_dtype, orr[8 * i + 4] * inv_l, orr[8 * i + 5] * inv_l),
                                       pack_16(P.out_dtype, orr[8 * i + 6] * inv_l, orr[8 * i + 7] * inv_l));
                }
            }
            fence_proxy_async_smem();
        }
        // every softmax thread reaches this barrier, also after a timeout (then nothing is stored)
        const int any_failed = named_bar_or(1, 128, ok ? 0 : 1);
        ok = !any_failed;
        if (!SPLIT && ok && warp == 2 && lane == 0) {
            const int n_blk = P.out_dtype == 0 ? 4 : 2, blk_cols = P.out_dtype == 0 ? 32 : 64;
            for (int kb = 0; kb < n_blk; ++kb) tma_store_4d(&tmO, base + kb * BLK_BYTES, kb * blk_cols, q0, h, b);
            tma_store_commit_and_wait_read();
        }
    }
    if (SPLIT) {
        // ------------------------------------------------------------------ the parts of the tile meet
        const int quad = warp & 3, row = quad * 32 + lane;
        const uint32_t o_row = tmem_base + ((uint32_t)(quad * 32) << 16) + PF_COL_O;
        __syncwarp();
        cluster_sync();  // every part has started, and its operand buffers are idle: its last MMA and its loads are over
        if (warp >= 2)
            for (int k = 0; k < parts; ++k) st_cluster_f2(map_to_cta(part_ml + part * 128 + row, (uint32_t)k), make_float2(m_ref, l));
        __syncwarp();
        cluster_sync();
        const int width = 128 / parts;  // columns a part finishes: 64, 32 or 16
        float f = 0.0f;                 // what this part's O is multiplied by
        if (warp >= 2) {
            float M = -INFINITY, L = 0.0f;
            for (int k = 0; k < parts; ++k) M = fmaxf(M, part_ml[k * 128 + row].x);
            for (int k = 0; k < parts; ++k) {
                const float2 ml = part_ml[k * 128 + row];
                if (ml.x != -INFINITY) L += ml.y * fast_exp2((ml.x - M) * m_unit);
            }
            // (a row no part saw a key for: L = 0, and 0 * inf = NaN as without parts)
            f = (m_ref == -INFINITY ? 0.0f : fast_exp2((m_ref - M) * m_unit)) * (1.0f / L);
            tc_fence_after();
        }
        auto scaled = [&](int col, float (&v)[16]) {  // 16 columns of this part's O, scaled; 0 (or NaN) where it saw no tile
            if (n_kv > 0) {
                tmem_ld16(o_row + col, *reinterpret_cast<uint32_t(*)[16]>(&v[0]));
                tc_wait_ld();
            } else {
#pragma unroll
                for (int i = 0; i < 16; ++i) v[i] = 0.0f;
            }
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] *= f;
        };
        if (warp >= 2 && ok)
            for (int col = 0; col < 128; col += 16) {
                const int owner = col / width;
                if (owner == part) continue;
                float v[16];
                scaled(col, v);
                const uint32_t dst = map_to_cta(base, (uint32_t)owner) + (uint32_t)(((part * width + col - owner * width) / 4 * 128 + row) * 16);
#pragma unroll
                for (int i = 0; i < 4; ++i) st_cluster_f4(dst + i * 128 * 16, make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]));
            }
        __syncwarp();
        cluster_sync();  // all columns have arrived, and none is on its way to a CTA that leaves
        if (warp >= 2 && ok)
            for (int c0 = 0; c0 < width; c0 += 16) {
                float own[16], sum[16];
                scaled(part * width + c0, own);
#pragma unroll
                for (int i = 0; i < 16; ++i) sum[i] = 0.0f;
                for (int k = 0; k < parts; ++k) {
                    const float4* src = reinterpret_cast<const float4*>(base) + (k * width + c0) / 4 * 128 + row;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float4 x = k == part ? make_float4(own[4 * i], own[4 * i + 1], own[4 * i + 2], own[4 * i + 3]) : src[i * 128];
                        sum[4 * i] += x.x; sum[4 * i + 1] += x.y; sum[4 * i + 2] += x.z; sum[4 * i + 3] += x.w;
                    }
                }
                if (q0 + row < P.Sq) {
                    const long long at = (long long)b * P.os[0] + (long long)h * P.os[1] + (long long)(q0 + row) * P.os[2] + part * width + c0;
                    if (P.out_dtype == 0) {
                        float4* o = reinterpret_cast<float4*>(static_cast<float*>(P.out) + at);
#pragma unroll
                        for (int i = 0; i < 4; ++i) o[i] = make_float4(sum[4 * i], sum[4 * i + 1], sum[4 * i + 2], sum[4 * i + 3]);
                    } else {
                        uint4* o = reinterpret_cast<uint4*>(static_cast<uint16_t*>(P.out) + at);
#pragma unroll
                        for (int i = 0; i < 2; ++i)
                            o[i] = make_uint4(pack_16(P.out_dtype, sum[8 * i], sum[8 * i + 1]), pack_16(P.out_dtype, sum[8 * i + 2], sum[8 * i + 3]),
                                              pack_16(P.out_dtype, sum[8 * i + 4], sum[8 * i + 5]), pack_16(P.out_dtype, sum[8 * i + 6], sum[8 * i + 7]));
                    }
                }
                __syncwarp();  // the next tcgen05.ld takes the whole warp
            }
    }
    // ---- teardown: every role falls through to here, also after a timeout
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, PF_TMEM_COLS);
    }
}

// V pre-pass: strided bf16 [B,Hkv,Skv,D] view -> contiguous f16 copy; raises *overflow when a value does not
// fit f16 (|v| > 65504, inf or NaN).  Thread 0 also clears the flag slot a later call will use.
struct CastVParams {
    const __nv_bfloat16* src;
    __half* dst;
    long long s0, s1, s2;  // element strides of batch, head, row
    int H, S, D;           // D is a multiple of 8
    long long n_vec;       // B*H*S*D / 8
    int* overflow;
    int* clear_slot;
};

__global__ void cast_v_to_f16_kernel(const CastVParams P) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *P.clear_slot = 0;
    const int vec_per_row = P.D / 8;
    bool bad = false;
    const long long stride = (long long)gridDim.x * blockDim.x;
    // four independent 16-byte loads per thread and trip: the pass is a plain stream and wants bytes in flight
    for (long long i0 = blockIdx.x * (long long)blockDim.x + threadIdx.x; i0 < P.n_vec; i0 += 4 * stride) {
        uint4 in[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const long long i = i0 + u * stride;
            if (i < P.n_vec) {
                const int c = (int)(i % vec_per_row);
                const long long row = i / vec_per_row;
                const int s = (int)(row % P.S);
                const int h = (int)((row / P.S) % P.H);
                const long long b = row / ((long long)P.S * P.H);
                in[u] = __ldg(reinterpret_cast<const uint4*>(P.src + b * P.s0 + h * P.s1 + s * P.s2 + c * 8));
            }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const long long i = i0 + u * stride;
            if (i < P.n_vec) {
                const __nv_bfloat162* iv = reinterpret_cast<const __nv_bfloat162*>(&in[u]);
                uint4 out;
                __half2* ov = reinterpret_cast<__half2*>(&out);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float2 f = __bfloat1622float2(iv[e]);
                    bad |= !(fabsf(f.x) <= 65504.0f) || !(fabsf(f.y) <= 65504.0f);
                    ov[e] = __floats2half2_rn(f.x, f.y);
                }
                *reinterpret_cast<uint4*>(P.dst + i * 8) = out;
            }
        }
    }
    if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicOr(P.overflow, 1);
}

}  // namespace fusor

// Attention for f32 tensors on warp-level bf16 MMAs, with the accuracy of f32 arithmetic.
//
// An f32 value is the exact sum of three bf16 terms, the first two rounded to nearest (cut off, every term has the value's sign,
// and what the product leaves out reaches 2^-21 of it, always to one side).  A product of two such sums is taken as six of its
// nine partial products; the three left out are at most 2^-23 of it and 2^-27 on average, to either side: the rounding of an f32
// product is 2^-24 at most and 2^-26 on average.  (Infinities and what rounds up to one: am_rows_f32.)  The warp MMA multiplies 1024 bf16 pairs per clock and SM, the FMA pipe
// 128 f32 pairs: with six products the MMA is ahead by a third, and it leaves the issue slots free for the softmax.
//
// One CTA = 64 query rows of one (batch, head), 4 warps x 16 rows.  K and V tiles arrive as f32 by cp.async in a staging
// buffer and are split by all threads into three bf16 planes each (rows padded by 16 bytes: no ldmatrix conflicts); the next
// tile's copy runs under the MMAs of this one.  Q is split once into planes of its own.
// B1 H32/8 S512 D64 causal: 35 us (62 us on the CUDA cores in general_attention_kernel); B2 H32/8 S2048 without a mask:
// 45 TFLOP/s at head_dim 64 and 44 at 128 (30 and 29), half of what the MMA pipe gives at six products; the staging and the
// split take most of the rest.  Error against 64 bits 0.39 to 0.86 times that of f32 arithmetic with its sums in order.
#pragma once
#include "attn_mma16.cuh"

namespace fusor {

template <int DP>
constexpr int a3_bn = DP <= 64 ? 64 : 32;  // keys per tile
template <int DP>
// Bytes of an f32 row.  The padding serves no access; without it two CTAs of head_dim 64 fit an SM, which was faster for full rows
// (B4 H16 S300 with a key mask 63.5 -> 54 us) and slower for few causal ones (B1 H32/8 S512 34.9 -> 38.5: heavy blocks pair up).
constexpr int a3_stage_pitch = DP * 4 + 16;
template <int DP>
constexpr size_t a3_smem_bytes = (size_t)am_pitch<DP> * 3 * (AM_BM + 2 * a3_bn<DP>) + (size_t)a3_stage_pitch<DP> * 2 * a3_bn<DP>;

// (x, y) -> three packed bf16 pairs whose sum is (x, y).  The first two are rounded to nearest, what is left then has at most 8
// significant bits.
__device__ __forceinline__ void split3(float x, float y, uint32_t (&t)[3]) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
        t[i] = *reinterpret_cast<const uint32_t*>(&h);
        x -= __uint_as_float(t[i] << 16);
        y -= __uint_as_float(t[i] & 0xffff0000u);
    }
    t[2] = __byte_perm(__float_as_uint(x), __float_as_uint(y), 0x7632);
}

// o = o alpha + t
template <int DP>
__device__ __forceinline__ void am_accumulate(float (&o)[DP / 8][4], const float (&t)[DP / 8][4], const float (&alpha)[2]) {
#pragma unroll
    for (int nd = 0; nd < DP / 8; ++nd)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const float2 x = ffma2(make_float2(o[nd][2 * r], o[nd][2 * r + 1]), make_float2(alpha[r], alpha[r]), make_float2(t[nd][2 * r], t[nd][2 * r + 1]));
            o[nd][2 * r] = x.x;
            o[nd][2 * r + 1] = x.y;
        }
}

template <int DP, bool ADD>
__global__ void __launch_bounds__(AM_THREADS, DP <= 64 ? 2 : 1) attn_mma32_kernel(const __grid_constant__ AttnMmaParams P) {
    extern __shared__ __align__(16) uint8_t am_smem[];
    constexpr int BN = a3_bn<DP>, PITCH = am_pitch<DP>, SP = a3_stage_pitch<DP>, CH = DP / 4;
    constexpr int QP = AM_BM * PITCH, KP = BN * PITCH;  // bytes of a plane
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t q_sm = smem_u32(am_smem), k_sm = q_sm + 3 * QP, v_sm = k_sm + 3 * KP, stage = v_sm + 3 * KP;
    uint8_t* stage_p = am_smem + (stage - q_sm);

    const int qt = P.n_q_tiles - 1 - (int)(blockIdx.x / (unsigned)(P.Hq * P.B));  // heavy (late) row blocks first
    const int hb = (int)(blockIdx.x % (unsigned)(P.Hq * P.B));
    const int h = hb % P.Hq, b = hb / P.Hq, hk = h / (P.Hq / P.Hkv);
    const int q0 = qt * AM_BM;
    const int offset = P.Skv - P.Sq;  // causal: key k allowed iff k <= q + offset
    const bool causal = P.mask_kind == 3 || P.mask_kind == 4;
    int k_begin = 0, k_end = P.Skv;
    if (causal) {
        k_end = min(P.Skv, min(q0 + AM_BM, P.Sq) + offset);
        if (P.mask_kind == 4) k_begin = max(0, q0 + offset - P.window + 1) / BN * BN;
    }
    const float* qg = static_cast<const float*>(P.q) + b * P.qs[0] + h * P.qs[1];
    const float* kg = static_cast<const float*>(P.k) + b * P.ks[0] + hk * P.ks[1];
    const float* vg = static_cast<const float*>(P.v) + b * P.vs[0] + hk * P.vs[1];

    auto load_rows = [&](uint32_t dst, const float* src, long long row_stride, int row0, int rows_end) {
#pragma unroll 8
        for (int i = tid; i < BN * CH; i += AM_THREADS) {
            const int r = i / CH, c = i % CH;
            const bool ok = row0 + r < rows_end && c * 4 < P.D;
            cp_async16_zfill(dst + r * SP + c * 16, src + (ok ? (long long)(row0 + r) * row_stride + c * 4 : 0), ok);
        }
    };
    // BN staged f32 rows -> rows of the three planes that start at dst (bytes from the start of shared memory)
    auto split_rows = [&](uint32_t dst, uint32_t plane, const uint8_t* src) {
#pragma unroll 4
        for (int i = tid; i < BN * CH / 2; i += AM_THREADS) {
            const int r = i / (CH / 2), c = i % (CH / 2);
            const float4 a = *reinterpret_cast<const float4*>(src + r * SP + c * 32), z = *reinterpret_cast<const float4*>(src + r * SP + c * 32 + 16);
            uint32_t t[4][3];
            split3(a.x, a.y, t[0]);
            split3(a.z, a.w, t[1]);
            split3(z.x, z.y, t[2]);
            split3(z.z, z.w, t[3]);
#pragma unroll
            for (int p = 0; p < 3; ++p)
                *reinterpret_cast<uint4*>(am_smem + dst + p * plane + r * PITCH + c * 16) = make_uint4(t[0][p], t[1][p], t[2][p], t[3][p]);
        }
    };
    for (int r = 0; r < AM_BM; r += BN) {
        load_rows(stage, qg, P.qs[2], q0 + r, P.Sq);
        cp_async_commit();
        cp_async_wait<0>();
        __syncthreads();
        split_rows(r * PITCH, QP, stage_p);
        __syncthreads();
    }
    load_rows(stage, kg, P.ks[2], k_begin, P.Skv);
    load_rows(stage + BN * SP, vg, P.vs[2], k_begin, P.Skv);
    cp_async_commit();

    const int r0 = q0 + warp * 16 + (lane >> 2);  // this thread's rows: r0 and r0 + 8
    const int cq = (lane & 3) * 2;                // column pair inside an 8-wide tile
    const int lm_j = lane >> 3, lm_r = lane & 7;
    const float c = P.scale * 1.4426950408889634f;  // scale > 0
    int first[2], last[2];            // keys each of the two rows may see
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int qi = r0 + r * 8;
        last[r] = causal ? min(P.Skv - 1, qi + offset) : P.Skv - 1;
        first[r] = P.mask_kind == 4 ? qi + offset - P.window + 1 : 0;
    }
    const float* mask0 = P.mask + (ADD ? (P.mask_kind == 1 ? (long long)min(r0, P.Sq - 1) : (long long)b) * P.ms[0] : 0);
    const long long mask_row8 = ADD && P.mask_kind == 1 ? (long long)(min(r0 + 8, P.Sq - 1) - min(r0, P.Sq - 1)) * P.ms[0] : 0;
    float o[DP / 8][4];
#pragma unroll
    for (int i = 0; i < DP / 8; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.0f;
    float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.0f, 0.0f};

    for (int kt = k_begin; kt < k_end; kt += BN) {
        cp_async_wait<0>();
        __syncthreads();  // the tile is staged, and everybody is done with the planes of the last one
        split_rows(3 * QP, KP, stage_p);
        split_rows(3 * QP + 3 * KP, KP, stage_p + BN * SP);
        __syncthreads();
        if (kt + BN < k_end) {
            load_rows(stage, kg, P.ks[2], kt + BN, P.Skv);
            load_rows(stage + BN * SP, vg, P.vs[2], kt + BN, P.Skv);
            cp_async_commit();
        }
        // ---- S = Q K^T.  The tensor core cuts off what lies below its running sum, so the five small partial products of
        // all of head_dim are summed before the large ones are added: only those DP / 16 steps lose anything.
        float s[BN / 8][4];
#pragma unroll
        for (int nt = 0; nt < BN / 8; ++nt) s[nt][0] = s[nt][1] = s[nt][2] = s[nt][3] = 0.0f;
        const uint32_t q_row = q_sm + (warp * 16 + (lm_j & 1) * 8 + lm_r) * PITCH + (lm_j >> 1) * 16;
        const uint32_t k_row = k_sm + ((lm_j >> 1) * 8 + lm_r) * PITCH + (lm_j & 1) * 16;
#pragma unroll
        for (int ks = 0; ks < DP / 16; ++ks) {
            uint32_t qa[3][4];
#pragma unroll
            for (int p = 0; p < 3; ++p) ldmatrix_x4(qa[p], q_row + p * QP + ks * 32);
#pragma unroll
            for (int np = 0; np < BN / 16; ++np) {  // two 8-key tiles
                uint32_t kf[3][4];
#pragma unroll
                for (int p = 0; p < 3; ++p) ldmatrix_x4(kf[p], k_row + p * KP + np * 16 * PITCH + ks * 32);
#pragma unroll
                for (int i = 2; i > 0; --i)  // partial products of terms (a, i - a)
#pragma unroll
                    for (int a = 0; a <= i; ++a) {
                        mma_16816<false>(s[2 * np], qa[a], kf[i - a][0], kf[i - a][1]);
                        mma_16816<false>(s[2 * np + 1], qa[a], kf[i - a][2], kf[i - a][3]);
                    }
            }
        }
#pragma unroll
        for (int ks = 0; ks < DP / 16; ++ks) {
            uint32_t qa[4];
            ldmatrix_x4(qa, q_row + ks * 32);
#pragma unroll
            for (int np = 0; np < BN / 16; ++np) {
                uint32_t kf[4];
                ldmatrix_x4(kf, k_row + np * 16 * PITCH + ks * 32);
                mma_16816<false>(s[2 * np], qa, kf[0], kf[1]);
                mma_16816<false>(s[2 * np + 1], qa, kf[2], kf[3]);
            }
        }
        // ---- additive masks (natural units), then the tile's edges (causal diagonal, window, past the last key)
        if (ADD) am_add_mask_tile<BN>(P, mask0, mask_row8, kt, cq, s);
        if (kt + BN > P.Skv || (causal && kt + BN - 1 > q0 + warp * 16 + offset) ||
            (P.mask_kind == 4 && kt <= q0 + warp * 16 + 15 + offset - P.window)) {
#pragma unroll
            for (int nt = 0; nt < BN / 8; ++nt)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int kj = kt + nt * 8 + cq + (e & 1);
                    if (kj > last[e >> 1] || kj < first[e >> 1]) s[nt][e] = -INFINITY;
                }
        }
        float alpha[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) am_softmax_row<BN, ADD, 0>(s, r, c, m[r], l[r], alpha[r]);
        // ---- O = O alpha + P V, the tile's product summed by itself (see attn_mma16.cuh)
        float t[DP / 8][4];
#pragma unroll
        for (int i = 0; i < DP / 8; ++i) t[i][0] = t[i][1] = t[i][2] = t[i][3] = 0.0f;
        uint32_t pa[BN / 16][3][4];
        const uint32_t v_row = v_sm + ((lm_j & 1) * 8 + lm_r) * PITCH + (lm_j >> 1) * 16;
#pragma unroll
        for (int kk = 0; kk < BN / 16; ++kk) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                uint32_t w[3];
                split3(s[2 * kk + (e >> 1)][2 * (e & 1)], s[2 * kk + (e >> 1)][2 * (e & 1) + 1], w);
                pa[kk][0][e] = w[0];
                pa[kk][1][e] = w[1];
                pa[kk][2][e] = w[2];
            }
#pragma unroll
            for (int nd = 0; nd < DP / 16; ++nd) {
                uint32_t vf[3][4];
#pragma unroll
                for (int p = 0; p < 3; ++p) ldmatrix_x4_trans(vf[p], v_row + p * KP + kk * 16 * PITCH + nd * 32);
#pragma unroll
                for (int i = 2; i > 0; --i)
#pragma unroll
                    for (int a = 0; a <= i; ++a) {
                        mma_16816<false>(t[2 * nd], pa[kk][a], vf[i - a][0], vf[i - a][1]);
                        mma_16816<false>(t[2 * nd + 1], pa[kk][a], vf[i - a][2], vf[i - a][3]);
                    }
            }
        }
#pragma unroll
        for (int kk = 0; kk < BN / 16; ++kk)
#pragma unroll
            for (int nd = 0; nd < DP / 16; ++nd) {
                uint32_t vf[4];
                ldmatrix_x4_trans(vf, v_row + kk * 16 * PITCH + nd * 32);
                mma_16816<false>(t[2 * nd], pa[kk][0], vf[0], vf[1]);
                mma_16816<false>(t[2 * nd + 1], pa[kk][0], vf[2], vf[3]);
            }
        am_accumulate<DP>(o, t, alpha);
    }
    am_store<DP, 0>(P, o, l, r0, cq, b, h);
}

}  // namespace fusor

// Attention on warp-level MMAs for 16-bit tensors that the tcgen05 kernels do not take (head_dim other than 128, or views
// that a TMA map cannot describe), with the accuracy of f32 arithmetic.
//
// The products q.k of 16-bit values are exact in f32, so S = Q K^T loses nothing on the tensor cores.  The softmax weights do
// not fit 16 bits: they are handed over as a sum of 16-bit terms, two for f16 (22 significant bits) and three for bf16 (24),
// each multiplied by the same V fragment.  f16 terms end at 2^-24, so f16 weights carry a factor of 2^14: what is lost of a weight
// is below 2^-39 of the row's largest.  (Without the factor, 2^-25: with 2047 keys 17.4 nats below one other their sum was off by
// 0.66 of itself, with it 3e-6.)  The tcgen05 kernels keep one 11-bit term; callers of this path had f32 arithmetic before
// (general_attention_kernel) and keep it.
//
// One CTA = 64 query rows of one (batch, head), 4 warps x 16 rows; K and V tiles of 64 keys come by cp.async into two
// buffers, rows padded by 16 bytes so that ldmatrix meets no bank conflict; Q stays in registers.  Three CTAs per SM
// (head_dim 64) hide each other's barriers and softmax.  Bound by the warp MMA pipe (538 TFLOP/s of bf16 products, measured):
// B4 H32/8 S2048 D64 causal 192 TFLOP/s in f16, three MMAs per useful two (four in bf16), 54 % of that pipe.
// Against the f32-arithmetic kernel that served these tensors: B8 H16 S300 D64 f16 with a key mask 852 -> 30 us, B2 H32/8 S1024
// D64 bf16 causal 2259 -> 64 us; error against 64 bits 0.38 to 0.98 times that of f32 arithmetic with its sums in order.
#pragma once
#include "ptx_sm100.cuh"

namespace fusor {

constexpr int AM_BM = 64, AM_BN = 64, AM_THREADS = 128;
constexpr int AM_F16_SHIFT = 14;  // 2^14 times a weight of at most 1 is far from the largest f16

struct AttnMmaParams {
    const void* q;
    const void* k;
    const void* v;
    void* out;
    const float* mask;
    int out_dtype;  // 0 = f32, 1 = bf16, 2 = f16
    int B, Hq, Hkv, Sq, Skv, D;
    long long qs[3], ks[3], vs[3], os[3];  // element strides of batch, head, row
    long long ms[2];                       // mask strides
    int mask_kind;                         // FUSOR_CUDA_MASK_*
    int window;
    int n_q_tiles;
    float scale;
};

__device__ __forceinline__ void cp_async16_zfill(uint32_t smem, const void* gmem, bool valid) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem), "l"(gmem), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// c (16x8, f32) += a (16x16, row) * b (16x8, col), both f16 or both bf16
template <bool F16>
__device__ __forceinline__ void mma_16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    if (F16)
        asm volatile(
            "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
            : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
            : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
    else
        mma_bf16_16816(c, a, b0, b1);
}

// Two f32 -> packed 16-bit pair; x and y keep what the pair does not hold.
template <bool F16>
__device__ __forceinline__ uint32_t split_pair(float& x, float& y) {
    uint32_t bits;
    float2 f;
    if (F16) {
        const __half2 h = __floats2half2_rn(x, y);
        bits = *reinterpret_cast<const uint32_t*>(&h);
        f = __half22float2(h);
    } else {
        const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
        bits = *reinterpret_cast<const uint32_t*>(&h);
        f = make_float2(__uint_as_float(bits << 16), __uint_as_float(bits & 0xffff0000u));
    }
    f = ffma2(f, make_float2(-1.0f, -1.0f), make_float2(x, y));
    x = f.x;
    y = f.y;
    return bits;
}

template <int DP>
constexpr int am_pitch = DP * 2 + 16;  // bytes of a row in shared memory
template <int DP>
constexpr size_t am_smem_bytes = (size_t)am_pitch<DP> * (AM_BM + 4 * AM_BN);

// s scale + mask with both steps rounded, as the composite computes it: next to a mask of -10000 the sum keeps 2^-11, and other
// roundings would show there
__device__ __forceinline__ void am_add_mask(float& s0, float& s1, float scale, float m0, float m1) {
    const float2 x = fadd2(fmul2(make_float2(s0, s1), make_float2(scale, scale)), make_float2(m0, m1));
    s0 = x.x;
    s1 = x.y;
}

// s scale + mask for a tile of BN keys from kt on: this thread's column pairs, by 8-byte loads at fixed offsets where the rows are
// contiguous, aligned and all there (B8 H16 S300 D64 f16 with a key mask 32.9 -> 30.4 us, bf16 37.0 -> 34.4: two 64-bit products
// and a clamp less per value), else value by value.  A key mask is the same for both rows of a thread (mask_row8 = 0).
template <int BN>
__device__ __forceinline__ void am_add_mask_tile(const AttnMmaParams& P, const float* mask0, long long mask_row8, int kt, int cq, float (&s)[BN / 8][4]) {
    const float* m = mask0 + kt + cq;
    if (P.ms[1] == 1 && kt + BN <= P.Skv && (reinterpret_cast<uintptr_t>(m) | (uintptr_t)(mask_row8 * 4)) % 8 == 0) {
#pragma unroll
        for (int nt = 0; nt < BN / 8; ++nt) {
            float2 x = __ldg(reinterpret_cast<const float2*>(m + nt * 8));
            am_add_mask(s[nt][0], s[nt][1], P.scale, x.x, x.y);
            if (mask_row8 != 0) x = __ldg(reinterpret_cast<const float2*>(m + nt * 8 + mask_row8));
            am_add_mask(s[nt][2], s[nt][3], P.scale, x.x, x.y);
        }
        return;
    }
#pragma unroll
    for (int nt = 0; nt < BN / 8; ++nt) {
        const int kj = kt + nt * 8 + cq;
        const float* k0 = mask0 + (long long)min(kj, P.Skv - 1) * P.ms[1];
        const float* k1 = mask0 + (long long)min(kj + 1, P.Skv - 1) * P.ms[1];
        float m0 = __ldg(k0), m1 = __ldg(k1);
        am_add_mask(s[nt][0], s[nt][1], P.scale, m0, m1);
        if (mask_row8 != 0) {
            m0 = __ldg(k0 + mask_row8);
            m1 = __ldg(k1 + mask_row8);
        }
        am_add_mask(s[nt][2], s[nt][3], P.scale, m0, m1);
    }
}

// Online softmax of row r (0 or 1) of the thread's fragment: a row lives in the four threads of a quad.  m is the row maximum,
// l this thread's part of the row sum.  s becomes the weights.  Without a mask tensor s holds raw products, c = scale log2(e)
// and m is in log2 units.  With one (ADD) s and m are in natural units and only differences are taken to log2: a finite mask
// value down to the lowest float stays finite, so that a row in which every key carries it is the mean of V and not NaN.
// SHIFT: weights and sums carry a factor of 2^SHIFT, which the division by l takes out again.
template <int BN, bool ADD, int SHIFT>
__device__ __forceinline__ void am_softmax_row(float (&s)[BN / 8][4], int r, float c, float& m, float& l, float& alpha) {
    constexpr float LOG2E = 1.4426950408889634f;
    float mx = fmaxf(s[0][2 * r], s[0][2 * r + 1]);
#pragma unroll
    for (int nt = 1; nt < BN / 8; ++nt) mx = fmax3(mx, s[nt][2 * r], s[nt][2 * r + 1]);
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
    mx = fmaxf(m, ADD ? mx : mx * c);
    // a row whose keys so far are all masked keeps m = -inf: subtract 0, so that its weights are 0 and not NaN
    const float ms = mx == -INFINITY ? 0.0f : mx;
    const float2 c2 = make_float2(c, c), e2 = make_float2(LOG2E, LOG2E), nm2 = make_float2(-ms, -ms);
    alpha = fast_exp2(ADD ? (m - ms) * LOG2E : m - ms);
    m = mx;
    float2 sum = make_float2(0.0f, 0.0f);
#pragma unroll
    for (int nt = 0; nt < BN / 8; ++nt) {
        const float2 sv = make_float2(s[nt][2 * r], s[nt][2 * r + 1]);
        const float2 x = ADD ? fmul2(fadd2(sv, nm2), e2) : ffma2(sv, c2, nm2);
        float2 p = make_float2(fast_exp2(x.x), fast_exp2(x.y));
        if (SHIFT) p = fmul2(p, make_float2(1 << SHIFT, 1 << SHIFT));  // (as a term of x it would cost the largest weights four bits)
        s[nt][2 * r] = p.x;
        s[nt][2 * r + 1] = p.y;
        sum = fadd2(sum, p);
    }
    l = l * alpha + (sum.x + sum.y);
}

// Rows of a warp's 16 (bits of `rows`) again, in plain f32 arithmetic: a lane owns a key of every 32 and, for O, the columns
// lane, lane + 32, ...  For operands that a sum of 16-bit terms does not stand for: next to an infinity its lower terms are zero or
// NaN, and the largest floats round up to one.  All of these leave a NaN behind, which is what sends a row here; one that is NaN
// by right (a NaN score) ends at its first tile.
template <int DT>  // 0 = f32, 1 = bf16, 2 = f16
__device__ __noinline__ void am_rows_f32(const AttnMmaParams& P, unsigned rows) {
    // (its place is worked out again: as arguments these values cost the main loop of the callers 7 %)
    const int hb = (int)(blockIdx.x % (unsigned)(P.Hq * P.B)), h = hb % P.Hq, b = hb / P.Hq;
    const int row0 = (P.n_q_tiles - 1 - (int)(blockIdx.x / (unsigned)(P.Hq * P.B))) * AM_BM + (int)(threadIdx.x >> 5) * 16;
    constexpr float LOG2E = 1.4426950408889634f;
    const int lane = threadIdx.x & 31, hk = h / (P.Hq / P.Hkv), offset = P.Skv - P.Sq;
    const bool causal = P.mask_kind == 3 || P.mask_kind == 4;
    for (; rows != 0; rows &= rows - 1) {
        const int qi = row0 + __ffs(rows) - 1;
        const int last = causal ? min(P.Skv - 1, qi + offset) : P.Skv - 1, first = P.mask_kind == 4 ? max(0, qi + offset - P.window + 1) : 0;
        const long long q_row = b * P.qs[0] + h * P.qs[1] + qi * P.qs[2], k_base = b * P.ks[0] + hk * P.ks[1], v_base = b * P.vs[0] + hk * P.vs[1];
        float m = -INFINITY, l = 0.0f, acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        for (int kt = first; kt <= last && l == l; kt += 32) {
            const int kj = kt + lane;
            float s = -INFINITY;
            if (kj <= last) {
                float dot = 0.0f;
                for (int d = 0; d < P.D; ++d) dot = fmaf(ld_as_float(P.q, DT, q_row + d), ld_as_float(P.k, DT, k_base + kj * P.ks[2] + d), dot);
                s = __fmul_rn(dot, P.scale);
                if (P.mask != nullptr) s = __fadd_rn(s, P.mask[(P.mask_kind == 1 ? qi : b) * P.ms[0] + kj * P.ms[1]]);
            }
            float mx = s;
#pragma unroll
            for (int i = 16; i > 0; i >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, i));
            mx = fmaxf(m, mx);
            const float ms = mx == -INFINITY ? 0.0f : mx, alpha = fast_exp2((m - ms) * LOG2E), p = fast_exp2((s - ms) * LOG2E);
            m = mx;
            float sum = p;
#pragma unroll
            for (int i = 16; i > 0; i >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, i);
            l = l * alpha + sum;
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[i] *= alpha;
            for (int j = 0; j < min(32, last + 1 - kt); ++j) {
                const float pj = __shfl_sync(0xffffffffu, p, j);
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (lane + 32 * i < P.D) acc[i] = fmaf(pj, ld_as_float(P.v, DT, v_base + (kt + j) * P.vs[2] + lane + 32 * i), acc[i]);
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (lane + 32 * i < P.D)
                st_from_float(P.out, P.out_dtype, b * P.os[0] + h * P.os[1] + qi * P.os[2] + lane + 32 * i, l == l ? acc[i] * (1.0f / l) : l);
    }
}

// O / l (a fully masked row gives 0 * inf = NaN, as the reference)
template <int DP, int DT>
__device__ __forceinline__ void am_store(const AttnMmaParams& P, const float (&o)[DP / 8][4], float (&l)[2], int r0, int cq, int b, int h) {
    unsigned again = 0;  // rows of the warp that hold a NaN although some key has weight
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        l[r] += __shfl_xor_sync(0xffffffffu, l[r], 1);
        l[r] += __shfl_xor_sync(0xffffffffu, l[r], 2);
        const int qi = r0 + r * 8;
        const float inv = 1.0f / l[r];
        const long long row = b * P.os[0] + h * P.os[1] + qi * P.os[2];
        bool nan = false;
#pragma unroll
        for (int nd = 0; nd < DP / 8; ++nd) {
            const int d = nd * 8 + cq;
            if (d >= P.D || qi >= P.Sq) continue;
            const float x = o[nd][2 * r] * inv, y = o[nd][2 * r + 1] * inv;
            nan = nan || x != x || y != y;
            if (P.out_dtype == 0) *reinterpret_cast<float2*>(static_cast<float*>(P.out) + row + d) = make_float2(x, y);
            else *reinterpret_cast<uint32_t*>(static_cast<uint16_t*>(P.out) + row + d) = pack_16(P.out_dtype, x, y);
        }
        unsigned lanes = __ballot_sync(0xffffffffu, nan && l[r] != 0.0f);
        for (; lanes != 0; lanes &= lanes - 1) again |= 1u << (r * 8 + ((__ffs(lanes) - 1) >> 2));
    }
    if (again != 0) {
        __syncwarp();  // the rows are stored again by other lanes
        am_rows_f32<DT>(P, again);
    }
}

// DP: head_dim rounded up to 32; columns D.. of Q, K and V read as zero
// ADD: an additive mask tensor is read
template <int DP, bool F16, bool ADD>
__global__ void __launch_bounds__(AM_THREADS, DP <= 64 ? 3 : 2) attn_mma16_kernel(const __grid_constant__ AttnMmaParams P) {
    extern __shared__ __align__(16) uint8_t am_smem[];
    constexpr int PITCH = am_pitch<DP>, CH = DP / 8;  // 16-byte chunks of a row
    constexpr int TERMS = F16 ? 2 : 3;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t q_sm = smem_u32(am_smem);
    const uint32_t kv_sm = q_sm + AM_BM * PITCH;  // [2 buffers]{K, V}

    // heavy (late) row blocks first
    const int qt = P.n_q_tiles - 1 - (int)(blockIdx.x / (unsigned)(P.Hq * P.B));
    const int hb = (int)(blockIdx.x % (unsigned)(P.Hq * P.B));
    const int h = hb % P.Hq, b = hb / P.Hq, hk = h / (P.Hq / P.Hkv);
    const int q0 = qt * AM_BM;
    const int offset = P.Skv - P.Sq;  // causal: key k allowed iff k <= q + offset
    const bool causal = P.mask_kind == 3 || P.mask_kind == 4;
    int k_begin = 0, k_end = P.Skv;
    if (causal) {
        k_end = min(P.Skv, min(q0 + AM_BM, P.Sq) + offset);
        if (P.mask_kind == 4) k_begin = max(0, q0 + offset - P.window + 1) / AM_BN * AM_BN;
    }
    const uint16_t* qg = static_cast<const uint16_t*>(P.q) + b * P.qs[0] + h * P.qs[1];
    const uint16_t* kg = static_cast<const uint16_t*>(P.k) + b * P.ks[0] + hk * P.ks[1];
    const uint16_t* vg = static_cast<const uint16_t*>(P.v) + b * P.vs[0] + hk * P.vs[1];

    auto load_rows = [&](uint32_t dst, const uint16_t* src, long long row_stride, int row0, int rows_end) {
#pragma unroll
        for (int i = tid; i < 64 * CH; i += AM_THREADS) {
            const int r = i / CH, c = i % CH;
            const bool ok = row0 + r < rows_end && c * 8 < P.D;
            cp_async16_zfill(dst + r * PITCH + c * 16, src + (ok ? (long long)(row0 + r) * row_stride + c * 8 : 0), ok);
        }
    };
    load_rows(q_sm, qg, P.qs[2], q0, P.Sq);
    load_rows(kv_sm, kg, P.ks[2], k_begin, P.Skv);
    load_rows(kv_sm + AM_BN * PITCH, vg, P.vs[2], k_begin, P.Skv);
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
    uint32_t qa[DP / 16][4];
    float o[DP / 8][4];
#pragma unroll
    for (int i = 0; i < DP / 8; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.0f;
    float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.0f, 0.0f};

    int buf = 0;
    for (int kt = k_begin; kt < k_end; kt += AM_BN, buf ^= 1) {
        cp_async_wait<0>();
        __syncthreads();  // the tile is here, and everybody is done with the other buffer
        if (kt + AM_BN < k_end) {
            const uint32_t nx = kv_sm + (buf ^ 1) * 2 * AM_BN * PITCH;
            load_rows(nx, kg, P.ks[2], kt + AM_BN, P.Skv);
            load_rows(nx + AM_BN * PITCH, vg, P.vs[2], kt + AM_BN, P.Skv);
            cp_async_commit();
        }
        if (kt == k_begin) {
#pragma unroll
            for (int ks = 0; ks < DP / 16; ++ks)
                ldmatrix_x4(qa[ks], q_sm + (warp * 16 + (lm_j & 1) * 8 + lm_r) * PITCH + (ks * 2 + (lm_j >> 1)) * 16);
        }
        const uint32_t kb = kv_sm + buf * 2 * AM_BN * PITCH, vb = kb + AM_BN * PITCH;
        // ---- S = Q K^T.  The tensor core cuts off what lies below its running sum, always towards zero, which shows against f32
        // arithmetic: half as many steps per sum, and the two halves added with rounding.
        float s[AM_BN / 8][4];
#pragma unroll
        for (int nt = 0; nt < AM_BN / 8; ++nt) {
            float odd[4] = {};
            s[nt][0] = s[nt][1] = s[nt][2] = s[nt][3] = 0.0f;
#pragma unroll
            for (int kp = 0; kp < DP / 32; ++kp) {
                uint32_t bf[4];
                ldmatrix_x4(bf, kb + (nt * 8 + lm_r) * PITCH + (kp * 4 + lm_j) * 16);
                mma_16816<F16>(s[nt], qa[2 * kp], bf[0], bf[1]);
                mma_16816<F16>(odd, qa[2 * kp + 1], bf[2], bf[3]);
            }
#pragma unroll
            for (int e = 0; e < 4; e += 2) {
                const float2 x = fadd2(make_float2(s[nt][e], s[nt][e + 1]), make_float2(odd[e], odd[e + 1]));
                s[nt][e] = x.x;
                s[nt][e + 1] = x.y;
            }
        }
        // ---- additive masks (natural units), then the tile's edges (causal diagonal, window, past the last key)
        if (ADD) am_add_mask_tile<AM_BN>(P, mask0, mask_row8, kt, cq, s);
        if (kt + AM_BN > P.Skv || (causal && kt + AM_BN - 1 > q0 + warp * 16 + offset) ||
            (P.mask_kind == 4 && kt <= q0 + warp * 16 + 15 + offset - P.window)) {
#pragma unroll
            for (int nt = 0; nt < AM_BN / 8; ++nt)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int kj = kt + nt * 8 + cq + (e & 1);
                    if (kj > last[e >> 1] || kj < first[e >> 1]) s[nt][e] = -INFINITY;
                }
        }
        // ---- online softmax
        float alpha[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) am_softmax_row<AM_BN, ADD, F16 ? AM_F16_SHIFT : 0>(s, r, c, m[r], l[r], alpha[r]);
        // ---- O = O alpha + P V.  For the same reason a tile's product is summed by itself, its first terms (four steps) apart from
        // the small ones (cut far below), and the sum over tiles is rounded.
        uint32_t pa[AM_BN / 16][TERMS][4];
#pragma unroll
        for (int kk = 0; kk < AM_BN / 16; ++kk)
#pragma unroll
            for (int i = 0; i < TERMS; ++i) {
                pa[kk][i][0] = split_pair<F16>(s[2 * kk][0], s[2 * kk][1]);
                pa[kk][i][1] = split_pair<F16>(s[2 * kk][2], s[2 * kk][3]);
                pa[kk][i][2] = split_pair<F16>(s[2 * kk + 1][0], s[2 * kk + 1][1]);
                pa[kk][i][3] = split_pair<F16>(s[2 * kk + 1][2], s[2 * kk + 1][3]);
            }
#pragma unroll
        for (int nd = 0; nd < DP / 16; ++nd) {
            float big[2][4] = {}, small[2][4] = {};
#pragma unroll
            for (int kk = 0; kk < AM_BN / 16; ++kk) {
                uint32_t bf[4];
                ldmatrix_x4_trans(bf, vb + (kk * 16 + (lm_j & 1) * 8 + lm_r) * PITCH + (nd * 2 + (lm_j >> 1)) * 16);
                mma_16816<F16>(big[0], pa[kk][0], bf[0], bf[1]);
                mma_16816<F16>(big[1], pa[kk][0], bf[2], bf[3]);
#pragma unroll
                for (int i = TERMS - 1; i > 0; --i) {
                    mma_16816<F16>(small[0], pa[kk][i], bf[0], bf[1]);
                    mma_16816<F16>(small[1], pa[kk][i], bf[2], bf[3]);
                }
            }
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    float* x = &o[2 * nd + j][2 * r];
                    const float2 y = fadd2(ffma2(make_float2(x[0], x[1]), make_float2(alpha[r], alpha[r]), make_float2(small[j][2 * r], small[j][2 * r + 1])),
                                           make_float2(big[j][2 * r], big[j][2 * r + 1]));
                    x[0] = y.x;
                    x[1] = y.y;
                }
        }
    }
    am_store<DP, F16 ? 2 : 1>(P, o, l, r0, cq, b, h);
}

}  // namespace fusor

// General attention kernel: f32 arithmetic on the CUDA cores, any head_dim <= 256, f32, bf16 or f16
// operands with arbitrary batch/head/row strides, additive mask tensors (QKMask, BatchKeyMask)
// or analytic causal / sliding-window masks.  It covers every call of the reference's
// Tensor::flash_attention (fusor-ml/fusor/src/composite/flash_attention.rs:52-73) that the
// tensor-core kernels do not take (f32 and 16-bit tensors of head_dim up to 128 in aligned views: attn_mma32, attn_mma16).
//
// Bound by the FMA pipe.  One CTA = 8 RT query rows of one (batch, head), 128 threads as 8 row groups x 16 columns: a thread
// owns RT rows (ty, ty + 8, ...) and, of each tile of 64 keys, the keys tx, tx + 16, tx + 32, tx + 48.  Q, K and V stand in
// shared memory as f32; S is summed in packed pairs along head_dim (even and odd elements apart), read with 16-byte loads:
// RT + 4 loads for 8 RT packed FMAs.  P goes through shared memory inside the warp that wrote it, and for O += P V the thread
// owns 4 neighbouring columns of every 64.  K of the next tile is fetched while P V runs, V of this one while S is summed.
// With one dot product per lane and key, four rows of a warp one after the other, H8 S1024 f32 took 1769 us at head_dim 192
// and 2284 at 256; now 330 and 461 (19 TFLOP/s; 30 at head_dim 64 and many rows, of 74 that the FMA pipe has).
#pragma once
#include "attn_mma16.cuh"
#include "ptx_sm100.cuh"

namespace fusor {

constexpr int GEN_BN = 64;       // keys per tile
constexpr int GEN_THREADS = 128;
constexpr int GEN_MAX_D = 256;
constexpr int GEN_P_PITCH = 80;  // floats; the two row groups of a warp write P to different banks

struct GeneralParams {
    const void* q;
    const void* k;
    const void* v;
    void* out;
    const float* mask;
    int q_dtype, k_dtype, v_dtype, out_dtype;  // 0 = f32, 1 = bf16, 2 = f16
    int B, Hq, Hkv, Sq, Skv, D;
    long long qs[3], ks[3], vs[3], os[3];  // element strides of batch, head, row
    long long ms[2];                       // mask strides
    int mask_kind;                         // FUSOR_CUDA_MASK_*
    int window;
    int n_q_tiles;
    float scale;
};

__host__ __device__ constexpr int gen_pitch(int D) { return (D + 3) / 4 * 4 + 4; }  // floats of a row of Q, K and V

// RT: query rows per thread.  NC: head_dim rounded up to 64 NC.  VEC: f32 operands whose rows allow 16-byte loads
// (cp.async); otherwise elements are read one by one and widened.
template <int RT, int NC, bool VEC>
__global__ void __launch_bounds__(GEN_THREADS) general_attention_kernel(const __grid_constant__ GeneralParams P) {
    extern __shared__ __align__(16) float gen_smem[];
    constexpr int BM = 8 * RT;
    constexpr float LOG2E = 1.4426950408889634f;
    const int pitch = gen_pitch(P.D), chunks = (P.D + 3) / 4;
    float* Qs = gen_smem;                   // [BM][pitch]
    float* Ks = Qs + BM * pitch;            // [GEN_BN][pitch]
    float* Vs = Ks + GEN_BN * pitch;        // [GEN_BN][pitch]
    float* Ps = Vs + GEN_BN * pitch;        // [BM][GEN_P_PITCH]

    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int qt = P.n_q_tiles - 1 - (int)(blockIdx.x / (unsigned)(P.Hq * P.B));  // heavy (late) row blocks first
    const int hb = (int)(blockIdx.x % (unsigned)(P.Hq * P.B));
    const int h = hb % P.Hq, b = hb / P.Hq, hk = h / (P.Hq / P.Hkv);
    const int q0 = qt * BM;
    const int offset = P.Skv - P.Sq;  // causal: key k allowed iff k <= q + offset
    const bool causal = P.mask_kind == 3 || P.mask_kind == 4;
    int k_begin = 0, k_end = P.Skv;
    if (causal) {
        k_end = min(P.Skv, min(q0 + BM, P.Sq) + offset);
        if (P.mask_kind == 4) k_begin = max(0, q0 + offset - P.window + 1) / GEN_BN * GEN_BN;
    }
    const long long qbase = b * P.qs[0] + h * P.qs[1], kbase = b * P.ks[0] + hk * P.ks[1], vbase = b * P.vs[0] + hk * P.vs[1];

    auto load = [&](float* dst, const void* src, int dtype, long long base, long long row_stride, int rows, int row0, int rows_end) {
        for (int i = tid; i < rows * chunks; i += GEN_THREADS) {
            const int r = i / chunks, c = (i - r * chunks) * 4;
            const bool ok = row0 + r < rows_end;
            const long long at = base + (ok ? (long long)(row0 + r) * row_stride + c : 0);
            float* d = dst + r * pitch + c;
            if (VEC) {
                cp_async16_zfill(smem_u32(d), static_cast<const float*>(src) + at, ok);
            } else {
                float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (ok) {
                    x.x = ld_as_float(src, dtype, at);
                    if (c + 1 < P.D) x.y = ld_as_float(src, dtype, at + 1);
                    if (c + 2 < P.D) x.z = ld_as_float(src, dtype, at + 2);
                    if (c + 3 < P.D) x.w = ld_as_float(src, dtype, at + 3);
                }
                *reinterpret_cast<float4*>(d) = x;
            }
        }
        if (VEC) cp_async_commit();
    };
    load(Qs, P.q, P.q_dtype, qbase, P.qs[2], BM, q0, P.Sq);
    load(Ks, P.k, P.k_dtype, kbase, P.ks[2], GEN_BN, k_begin, P.Skv);

    float m[RT], l[RT];
    float2 o[RT][2 * NC];
#pragma unroll
    for (int r = 0; r < RT; ++r) {
        m[r] = -INFINITY;
        l[r] = 0.0f;
#pragma unroll
        for (int i = 0; i < 2 * NC; ++i) o[r][i] = make_float2(0.0f, 0.0f);
    }

    for (int kt = k_begin; kt < k_end; kt += GEN_BN) {
        if (VEC) cp_async_wait<0>();
        __syncthreads();  // K of this tile is here; everybody is done with V of the last one
        load(Vs, P.v, P.v_dtype, vbase, P.vs[2], GEN_BN, kt, P.Skv);
        // ---- S = Q K^T
        float2 acc[RT][4];
#pragma unroll
        for (int r = 0; r < RT; ++r)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[r][j] = make_float2(0.0f, 0.0f);
        const float* qr = Qs + ty * pitch;
        const float* kr = Ks + tx * pitch;
#pragma unroll 2
        for (int d = 0; d < chunks * 4; d += 4) {
            float4 kv[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) kv[j] = *reinterpret_cast<const float4*>(kr + j * 16 * pitch + d);
#pragma unroll
            for (int r = 0; r < RT; ++r) {
                const float4 qv = *reinterpret_cast<const float4*>(qr + r * 8 * pitch + d);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    acc[r][j] = ffma2(make_float2(qv.x, qv.y), make_float2(kv[j].x, kv[j].y), acc[r][j]);
                    acc[r][j] = ffma2(make_float2(qv.z, qv.w), make_float2(kv[j].z, kv[j].w), acc[r][j]);
                }
            }
        }
        // ---- scale, mask, online softmax, in natural units: only differences are taken to log2, so that finite mask values down
        // to the lowest float stay finite
        const bool edge = kt + GEN_BN > P.Skv || (causal && kt + GEN_BN - 1 > q0 + offset) || (P.mask_kind == 4 && kt <= q0 + BM - 1 + offset - P.window);
        __syncwarp();  // the warp has read the P rows of the last tile
#pragma unroll
        for (int r = 0; r < RT; ++r) {
            const int qi = q0 + ty + 8 * r;
            float s[4], mx = m[r];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int kj = kt + tx + 16 * j;
                s[j] = __fmul_rn(acc[r][j].x + acc[r][j].y, P.scale);
                if (P.mask != nullptr) {
                    const long long row = P.mask_kind == 1 ? min(qi, P.Sq - 1) : b;
                    s[j] = __fadd_rn(s[j], __ldg(P.mask + row * P.ms[0] + (long long)min(kj, P.Skv - 1) * P.ms[1]));  // rounded as the composite does
                }
                if (edge && (kj >= P.Skv || (causal && kj > qi + offset) || (P.mask_kind == 4 && kj <= qi + offset - P.window))) s[j] = -INFINITY;
                mx = fmaxf(mx, s[j]);
            }
#pragma unroll
            for (int i = 8; i > 0; i >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, i));
            // a row whose keys so far are all masked keeps m = -inf: subtract 0, so that its weights are 0 and not NaN
            const float ms = mx == -INFINITY ? 0.0f : mx;
            const float alpha = fast_exp2((m[r] - ms) * LOG2E);
            m[r] = mx;
            float sum = 0.0f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float p = fast_exp2((s[j] - ms) * LOG2E);
                sum += p;
                Ps[(ty + 8 * r) * GEN_P_PITCH + tx + 16 * j] = p;
            }
            l[r] = l[r] * alpha + sum;
#pragma unroll
            for (int i = 0; i < 2 * NC; ++i) o[r][i] = fmul2(o[r][i], make_float2(alpha, alpha));
        }
        if (VEC) cp_async_wait<0>();
        __syncthreads();  // V is here; everybody is done with K
        if (kt + GEN_BN < k_end) load(Ks, P.k, P.k_dtype, kbase, P.ks[2], GEN_BN, kt + GEN_BN, P.Skv);
        // ---- O += P V
        const float* pr = Ps + ty * GEN_P_PITCH;
#pragma unroll 2
        for (int j0 = 0; j0 < GEN_BN; j0 += 4) {
            float4 p[RT];
#pragma unroll
            for (int r = 0; r < RT; ++r) p[r] = *reinterpret_cast<const float4*>(pr + r * 8 * GEN_P_PITCH + j0);
#pragma unroll
            for (int jj = 0; jj < 4; ++jj) {
#pragma unroll
                for (int n = 0; n < NC; ++n) {
                    // columns past the row's end belong to no output: their sums are never stored
                    const int col = n * 64 + tx * 4;
                    const float4 v = *reinterpret_cast<const float4*>(Vs + (j0 + jj) * pitch + (col < pitch ? col : 0));
#pragma unroll
                    for (int r = 0; r < RT; ++r) {
                        const float pj = jj == 0 ? p[r].x : jj == 1 ? p[r].y : jj == 2 ? p[r].z : p[r].w;
                        o[r][2 * n] = ffma2(make_float2(pj, pj), make_float2(v.x, v.y), o[r][2 * n]);
                        o[r][2 * n + 1] = ffma2(make_float2(pj, pj), make_float2(v.z, v.w), o[r][2 * n + 1]);
                    }
                }
            }
        }
    }
    const long long obase = b * P.os[0] + h * P.os[1];
#pragma unroll
    for (int r = 0; r < RT; ++r) {
#pragma unroll
        for (int i = 8; i > 0; i >>= 1) l[r] += __shfl_xor_sync(0xffffffffu, l[r], i);
        const int qi = q0 + ty + 8 * r;
        if (qi >= P.Sq) continue;
        const float inv = 1.0f / l[r];  // fully masked row: 0 * inf = NaN, as the reference
        const long long row = obase + (long long)qi * P.os[2];
#pragma unroll
        for (int n = 0; n < NC; ++n) {
            const int d = n * 64 + tx * 4;
            const float2 a = fmul2(o[r][2 * n], make_float2(inv, inv)), z = fmul2(o[r][2 * n + 1], make_float2(inv, inv));
            if (VEC && P.out_dtype == 0) {
                if (d < P.D) *reinterpret_cast<float4*>(static_cast<float*>(P.out) + row + d) = make_float4(a.x, a.y, z.x, z.y);
                continue;
            }
            if (d < P.D) st_from_float(P.out, P.out_dtype, row + d, a.x);
            if (d + 1 < P.D) st_from_float(P.out, P.out_dtype, row + d + 1, a.y);
            if (d + 2 < P.D) st_from_float(P.out, P.out_dtype, row + d + 2, z.x);
            if (d + 3 < P.D) st_from_float(P.out, P.out_dtype, row + d + 3, z.y);
        }
    }
}

inline size_t general_smem_bytes(int D, int rt) {
    return sizeof(float) * (size_t)((8 * rt + 2 * GEN_BN) * gen_pitch(D) + 8 * rt * GEN_P_PITCH);
}

}  // namespace fusor

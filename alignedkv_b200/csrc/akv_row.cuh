// Pieces of a (batch, query head) row shared by the decode step (akv_decode.cu) and the operator classes' entry points
// (akv_operators.cu): the residual tokens' scores and the magnitude probe.
#pragma once
#include "akv_common.cuh"

namespace akv {

constexpr int TOPK = 32;     // residue classes of the magnitude probe (extension/v_cache_file.py:16)
constexpr int BLK = 64;      // tokens per K block (extension/k_cache_file.py:5-6)

// Score of one residual token of a (batch, query head) row by four threads: thread % 4 = quarter of the channels in 16-byte
// pieces, all loads of a row in flight at once, fp32 dot product rounded to fp16, then divided by sqrt(D) and rounded again,
// which is what `matmul(q, restk^T) / sqrt(D)` on fp16 tensors produces (k_cache_file.py:156-157).  kr: the token's key, or null.
// All four threads return it.
__device__ __forceinline__ __half residual_score_of(const __half* __restrict__ qr, const __half* __restrict__ kr, int D, float sqrt_d) {
    const int c = threadIdx.x & 3;
    float acc = 0.f;
    if (kr) {
#pragma unroll 4
        for (int d = c * 8; d < D; d += 32) {
            const uint4 kv = *reinterpret_cast<const uint4*>(kr + d), qv = *reinterpret_cast<const uint4*>(qr + d);
            const __half2* k2 = reinterpret_cast<const __half2*>(&kv);
            const __half2* q2 = reinterpret_cast<const __half2*>(&qv);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float2 kf = __half22float2(k2[i]), qf = __half22float2(q2[i]);
                acc = fmaf(qf.x, kf.x, acc);
                acc = fmaf(qf.y, kf.y, acc);
            }
        }
    }
    acc += __shfl_xor_sync(0xFFFFFFFFu, acc, 1);
    acc += __shfl_xor_sync(0xFFFFFFFFu, acc, 2);
    return __float2half_rn(__half2float(__float2half_rn(acc)) / sqrt_d);
}
// ... of residual token tid / 4 of a row, by 256 threads, 0 <= tid / 4 < rest <= 64
__device__ __forceinline__ __half residual_score(const __half* __restrict__ qr, const __half* __restrict__ restk, int b, int h,
                                                 int H, int D, int rest, float sqrt_d, bool wanted) {
    const int r = threadIdx.x >> 2;
    return residual_score_of(qr, wanted && r < rest ? restk + (((size_t)b * BLK + r) * H + h) * D : nullptr, D, sqrt_d);
}
// The same for a CTA of 256 threads, written into the row; only tokens with t_lo <= qn + r < t_hi (a row split across CTAs).
__device__ __forceinline__ void residual_scores(uint16_t* __restrict__ row, const __half* __restrict__ qr,
                                                const __half* __restrict__ restk, int b, int h, int H, int D, int qn,
                                                int rest, float sqrt_d, int t_lo, int t_hi) {
    const int r = threadIdx.x >> 2;
    const bool mine = r < rest && qn + r >= t_lo && qn + r < t_hi;
    const __half v = residual_score(qr, restk, b, h, H, D, rest, sqrt_d, mine);
    if (mine && (threadIdx.x & 3) == 0) row[qn + r] = __half_as_ushort(v);
}

// Magnitude probe of a row by a CTA of NT threads: o_test[d] = sum_j |half((first_8[row_j][d] << 8) + 0x80)| * p_j over the
// class maxima (V_cache.cu:104-119), p_j = key[0][j] (fp16 bits), rows row_j = key[1][j] * 32 + j, accumulated in fp16 in j
// order.  F = high bytes of the row's KV head.  The rows are gathered by the whole CTA, 16 bytes a thread (all 32 rows of 128
// bytes in one load), 256 channels at a time.
template <int NT>
__device__ __forceinline__ void probe_row(const uint8_t* __restrict__ F, const uint32_t (*key)[TOPK], uint8_t (*rows)[256],
                                          uint32_t* __restrict__ out, int max_seq_len, int D) {
    const int tid = threadIdx.x;
    const bool vec = (reinterpret_cast<uintptr_t>(F) & 15u) == 0;
    for (int d0 = 0; d0 < D; d0 += 256) {
        const int dn = min(256, D - d0);
        if (d0 > 0) __syncthreads();
        auto src = [&](int j) { return F + (size_t)min((int)key[1][j] * TOPK + j, max_seq_len - 1) * D + d0; };
        if (vec) {
            const int per = dn >> 4;                             // 16-byte pieces of a row (D is a multiple of 64)
            for (int i = tid; i < TOPK * per; i += NT)
                *reinterpret_cast<uint4*>(&rows[i / per][16 * (i % per)]) = __ldg(reinterpret_cast<const uint4*>(src(i / per)) + i % per);
        } else {
            const int per = dn >> 1;
            for (int i = tid; i < TOPK * per; i += NT)
                *reinterpret_cast<uint16_t*>(&rows[i / per][2 * (i % per)]) = __ldg(reinterpret_cast<const uint16_t*>(src(i / per)) + i % per);
        }
        __syncthreads();
        for (int c = tid; 2 * c < dn; c += NT) {
            uint32_t acc = 0;
#pragma unroll 8
            for (int j = 0; j < TOPK; ++j) {
                const uint32_t f = *reinterpret_cast<const uint16_t*>(&rows[j][2 * c]);
                acc = hfma2_bits(__byte_perm(f, 0x80u, 0x1404) & 0x7FFF7FFFu, key[0][j] | (key[0][j] << 16), acc);
            }
            out[(d0 >> 1) + c] = acc;
        }
    }
}

}  // namespace akv

// What K_Cache_Class.decoding_compute and V_Cache_Class.decoding_compute do for one decode token, as two library calls:
// the tensor operations around the streaming kernels (extension/k_cache_file.py:132-159, extension/v_cache_file.py:119-190)
// in one small kernel each.
//   akv_k_scores   operator_prologue_kernel (alignment inputs, residual tokens' scores, -inf padding), q.K^T
//   akv_v_output   operator_probe_kernel (class maxima, magnitude probe, residual tokens' part of the output), P.V
// As tensor operations these are 24 launches and 315 us per token at batch 4 x 32 heads x 2085 tokens, most of it the host's.
#include "akv_row.cuh"

namespace akv {

int launch_k_compute(const uint8_t*, const uint8_t*, const uint8_t*, const uint8_t*, const uint8_t*, const uint8_t*, uint8_t*,
                     int, int, int, int, int, int, int, float, int, cudaStream_t);
bool v_compute_takes_probe(const uint8_t*, const uint8_t*, const uint8_t*, const uint8_t*, const uint8_t*, int, int, int, int);
bool v_compute_adds_residual(const uint8_t*, const uint8_t*, const uint8_t*, const uint8_t*, const uint8_t*, int, int, int,
                             int, int, int, int);
int launch_v_compute_res(const uint8_t*, const uint8_t*, const uint8_t*, const uint8_t*, uint8_t*, const uint8_t*,
                         const uint8_t*, const uint8_t*, uint8_t*, int, int, int, int, int, int, int, int, int, cudaStream_t);

namespace {

size_t align_up(size_t x) { return (x + 255) & ~(size_t)255; }

// One CTA per (batch, head).  Exponent upper bounds of the products q_d * k_{t,d} and their maximum
// (extension/k_cache_file.py:136-138), scores of the residual tokens (:156-157), -inf behind them (:158).
__global__ void __launch_bounds__(256)
operator_prologue_kernel(const uint16_t* __restrict__ q, const uint16_t* __restrict__ k_exp, const __half* __restrict__ restk,
                         uint16_t* __restrict__ kq, uint8_t* __restrict__ kqmax, uint16_t* __restrict__ s, int H, int D, int R,
                         int qn, int rest, float sqrt_d) {
    __shared__ uint32_t red[8];
    pdl_enter();
    const int bh = blockIdx.x, b = bh / H, h = bh - b * H, tid = threadIdx.x;
    uint32_t m = 0;
    for (int c = tid; c < (D >> 1); c += 256) {
        const uint32_t w = reinterpret_cast<const uint32_t*>(q)[(size_t)bh * (D >> 1) + c];
        const uint32_t e = ((w >> 10) & 0x1Fu) | (((w >> 26) & 0x1Fu) << 8);
        const uint32_t x = __vadd4(e, k_exp[(size_t)bh * (D >> 1) + c]) & 0xFFFFu;      // bytewise, modulo 256
        kq[(size_t)bh * (D >> 1) + c] = (uint16_t)x;
        m = max(m, max(x & 0xFFu, x >> 8));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xFFFFFFFFu, m, o));
    if ((tid & 31) == 0) red[tid >> 5] = m;
    uint16_t* row = s + (size_t)bh * R;
    residual_scores(row, reinterpret_cast<const __half*>(q) + (size_t)bh * D, restk, b, h, H, D, qn, rest, sqrt_d, 0, qn + rest);
    for (int t = qn + rest + tid; t < R; t += 256) row[t] = 0xFC00u;
    __syncthreads();
    if (tid == 0) {
#pragma unroll
        for (int i = 1; i < 8; ++i) m = max(m, red[i]);
        kqmax[bh] = (uint8_t)m;
    }
}

// fp16 bits as torch.max orders them (NaN above everything, -0 equal to +0), in 16 bits
__device__ __forceinline__ uint32_t order16(uint32_t x) {
    if ((x & 0x7FFFu) > 0x7C00u) return 0xFFFFu;
    if (x == 0x8000u) x = 0;
    return x & 0x8000u ? 0xFFFFu & ~x : x | 0x8000u;
}

// One CTA per (batch, head): the largest probability of each residue class modulo 32 with its first position
// (extension/v_cache_file.py:128-130), the probe over them, and half(sum_r p[qn + r] * restv[r]) (:189) into res (rest > 0).
// The probabilities are the caller's, any fp16 value.  Bound by latency: the row's loads in flight together, one reduction,
// one gather, the chain of 32 additions.
constexpr int PROBE_NT = 256;
__global__ void __launch_bounds__(PROBE_NT)
operator_probe_kernel(const uint16_t* __restrict__ s, const uint8_t* __restrict__ first8, const __half* __restrict__ restv,
                      uint16_t* __restrict__ test_o, uint16_t* __restrict__ res, int max_seq_len, int H, int D, int s_row, int qn,
                      int rest) {
    constexpr int NT = PROBE_NT, NW = NT / 32;
    __shared__ __align__(16) uint32_t key[NW][TOPK];
    __shared__ __align__(16) uint8_t rows[TOPK][256];
    __shared__ float part[4][256];
    pdl_turn();
    const int bh = blockIdx.x, b = bh / H, h = bh - b * H;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint16_t* row = s + (size_t)bh * s_row;
    // a thread's vectors of 8 all have the same eight classes (8 (tid % 4) + 0..7)
    uint32_t best[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) best[j] = 0;
#pragma unroll 4
    for (int v = tid; v < (qn >> 3); v += NT) {
        const uint4 w = __ldg(reinterpret_cast<const uint4*>(row) + v);
        const uint32_t at = 0xFFFFu - (uint32_t)(v >> 2);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint32_t x = u4w(w, j);
            best[2 * j] = max(best[2 * j], order16(x & 0xFFFFu) << 16 | at);
            best[2 * j + 1] = max(best[2 * j + 1], order16(x >> 16) << 16 | at);
        }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) best[j] = max(best[j], __shfl_xor_sync(0xFFFFFFFFu, best[j], o));
    if (lane < 4) {
        *reinterpret_cast<uint4*>(&key[warp][8 * lane]) = make_uint4(best[0], best[1], best[2], best[3]);
        *reinterpret_cast<uint4*>(&key[warp][8 * lane + 4]) = make_uint4(best[4], best[5], best[6], best[7]);
    }
    __syncthreads();
    if (tid < TOPK) {
        uint32_t k = key[0][tid];
        for (int i = 1; i < NW; ++i) k = max(k, key[i][tid]);
        const uint32_t at = 0xFFFFu - (k & 0xFFFFu);
        key[1][tid] = at;
        key[0][tid] = row[at * TOPK + tid];                      // (qn is a positive multiple of 64: every class has a position)
    }
    __syncthreads();
    const int hd = D >> 1;
    probe_row<NT>(first8 + (size_t)bh * max_seq_len * D, key, rows, reinterpret_cast<uint32_t*>(test_o) + (size_t)bh * hd,
                  max_seq_len, D);
    if (rest == 0) return;                                       // (uniform)
    // item = (channel pair, share g of the tokens), fp32 sums, the shares added in order (D <= 256)
    for (int i = tid; i < 4 * hd; i += NT) {
        const int g = i / hd, c = i - g * hd;
        const __half* vr = restv + ((size_t)b * BLK * H + h) * D + 2 * c;
        float a0 = 0.f, a1 = 0.f;
#pragma unroll 8
        for (int r = g; r < rest; r += 4) {
            const float2 f = __half22float2(*reinterpret_cast<const __half2*>(vr + (size_t)r * H * D));
            const float pv = __half2float(__ushort_as_half(row[qn + r]));
            a0 = fmaf(pv, f.x, a0);
            a1 = fmaf(pv, f.y, a1);
        }
        part[g][2 * c] = a0;
        part[g][2 * c + 1] = a1;
    }
    __syncthreads();
    for (int d = tid; d < D; d += NT)
        res[(size_t)bh * D + d] = __half_as_ushort(__float2half_rn(((part[0][d] + part[1][d]) + part[2][d]) + part[3][d]));
}

// out = half(out + res), for the P.V forms that do not add it themselves (all planes read).
__global__ void __launch_bounds__(256)
operator_add_kernel(uint16_t* __restrict__ out, const uint16_t* __restrict__ res, int n) {
    pdl_enter();
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i < n)
        out[i] = __half_as_ushort(__float2half_rn(__half2float(__ushort_as_half(out[i])) + __half2float(__ushort_as_half(res[i]))));
}

// Threshold bytes (extension/v_cache_file.py:142,156-160), for the P.V forms that do not derive them: a warp per row.
__global__ void __launch_bounds__(128)
operator_threshold_kernel(const uint16_t* __restrict__ test_o, const uint8_t* __restrict__ v_exp, uint8_t* __restrict__ amin,
                          int rows, int H, int D) {
    pdl_enter();
    const int i = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (i >= rows) return;
    const uint32_t m = v_threshold_warp(test_o, v_exp, i, H, 1, D, lane);
    if (lane == 0) amin[i] = (uint8_t)m;
}

}  // namespace
}  // namespace akv

using namespace akv;

extern "C" {

long long akv_operator_scratch_bytes(int bsz, int n_heads, int head_dim) {
    if (bsz <= 0 || n_heads <= 0 || head_dim <= 0) return -1;
    const size_t rows = (size_t)bsz * n_heads;
    return (long long)(2 * align_up(rows * head_dim * 2) + align_up(rows));
}

int akv_k_scores(const void* k_first_8, const void* k_mid_4, const void* k_last_4, const void* k_exp_max, const void* restk,
                 const void* q, void* s, void* scratch, long long scratch_bytes, int bsz, int n_heads, int n_blocks,
                 int n_max_blocks, int head_dim, int rest_len, float inv_sqrt_dim, int reference, void* stream) {
    set_error("");
    const int B = bsz, H = n_heads, D = head_dim;
    AKV_REQUIRE(k_first_8 && k_mid_4 && k_last_4 && k_exp_max && restk && q && s && scratch, AKV_ERR_NULL,
                "k_scores: null pointer");
    AKV_REQUIRE(B > 0 && H > 0 && D > 0 && D % 64 == 0 && D <= 1024 && n_blocks >= 0 && n_blocks <= n_max_blocks &&
                rest_len >= 0 && rest_len <= BLK, AKV_ERR_SHAPE, "k_scores: unsupported extent (bsz %d, heads %d, head_dim %d "
                "[multiple of 64], blocks %d of %d, residual tokens %d)", B, H, D, n_blocks, n_max_blocks, rest_len);
    AKV_REQUIRE(scratch_bytes >= akv_operator_scratch_bytes(B, H, D), AKV_ERR_SHAPE,
                "k_scores: scratch of %lld bytes is too small", scratch_bytes);
    AKV_REQUIRE(aligned16(k_exp_max) && aligned16(restk) && aligned16(q) && aligned16(s) && aligned16(scratch), AKV_ERR_ALIGN,
                "k_scores: pointers must be 16-byte aligned");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    uint8_t* kq = static_cast<uint8_t*>(scratch);
    uint8_t* kqmax = kq + align_up((size_t)B * H * D);
    const int R = (n_blocks + 1) * BLK;
    launch_chained(operator_prologue_kernel, dim3(B * H), dim3(256), 0, st, static_cast<const uint16_t*>(q),
                   static_cast<const uint16_t*>(k_exp_max), static_cast<const __half*>(restk), reinterpret_cast<uint16_t*>(kq),
                   kqmax, static_cast<uint16_t*>(s), H, D, R, n_blocks * BLK, rest_len, sqrtf((float)D));
    const int rc = cuda_status(cudaGetLastError(), "k_scores launch");
    if (rc != AKV_OK || n_blocks == 0) return rc;
    return launch_k_compute(static_cast<const uint8_t*>(k_first_8), static_cast<const uint8_t*>(k_mid_4),
                            static_cast<const uint8_t*>(k_last_4), kq, kqmax, static_cast<const uint8_t*>(q),
                            static_cast<uint8_t*>(s), B, H, 1, n_blocks, n_max_blocks, D, BLK, inv_sqrt_dim, reference, st);
}

int akv_v_output(const void* v_first_8, const void* v_mid_4, const void* v_last_4, const void* v_exp_max, const void* restv,
                 const void* s, void* out, void* scratch, long long scratch_bytes, int bsz, int n_heads, int max_seq_len,
                 int head_dim, int s_last_dim, int n, int rest_len, int reference, void* stream) {
    set_error("");
    const int B = bsz, H = n_heads, D = head_dim, rows = B * H;
    AKV_REQUIRE(v_first_8 && v_mid_4 && v_last_4 && v_exp_max && restv && s && out && scratch, AKV_ERR_NULL,
                "v_output: null pointer");
    // (positions of the class maxima are kept in 16 bits)
    AKV_REQUIRE(B > 0 && H > 0 && D > 0 && D % 64 == 0 && D <= 256 && n > 0 && n % BLK == 0 && n <= max_seq_len &&
                n <= 32 * 65536 && rest_len >= 0 && rest_len <= BLK && s_last_dim % 8 == 0 && n + rest_len <= s_last_dim,
                AKV_ERR_SHAPE, "v_output: unsupported extent (bsz %d, heads %d, head_dim %d [multiple of 64, at most 256], %d + "
                "%d tokens of %d, rows of %d)", B, H, D, n, rest_len, max_seq_len, s_last_dim);
    AKV_REQUIRE((long long)B * H * D < (1ll << 31), AKV_ERR_OVERFLOW, "v_output: too many rows");
    AKV_REQUIRE(scratch_bytes >= akv_operator_scratch_bytes(B, H, D), AKV_ERR_SHAPE,
                "v_output: scratch of %lld bytes is too small", scratch_bytes);
    AKV_REQUIRE(aligned16(v_first_8) && aligned16(v_mid_4) && aligned16(v_last_4) && aligned16(v_exp_max) && aligned16(restv) &&
                aligned16(s) && aligned16(out) && aligned16(scratch), AKV_ERR_ALIGN, "v_output: pointers must be 16-byte aligned");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const size_t part = align_up((size_t)rows * D * 2);
    uint8_t* test_o = static_cast<uint8_t*>(scratch);
    uint8_t* res = test_o + part;
    uint8_t* amin = res + part;
    const uint8_t *f8 = static_cast<const uint8_t*>(v_first_8), *m4 = static_cast<const uint8_t*>(v_mid_4),
                  *l4 = static_cast<const uint8_t*>(v_last_4), *ve = static_cast<const uint8_t*>(v_exp_max),
                  *sp = static_cast<const uint8_t*>(s);
    uint8_t* o = static_cast<uint8_t*>(out);
    launch_chained(operator_probe_kernel, dim3(rows), dim3(PROBE_NT), 0, st, static_cast<const uint16_t*>(s), f8,
                   static_cast<const __half*>(restv), reinterpret_cast<uint16_t*>(test_o), reinterpret_cast<uint16_t*>(res),
                   max_seq_len, H, D, s_last_dim, n, rest_len);
    int rc = cuda_status(cudaGetLastError(), "v_output probe launch");
    if (rc != AKV_OK) return rc;
    const bool takes_probe = v_compute_takes_probe(f8, m4, l4, sp, o, 1, D, s_last_dim, n);
    const bool adds = rest_len > 0 && v_compute_adds_residual(f8, m4, l4, sp, o, B, H, 1, D, s_last_dim, n, reference);
    if (!takes_probe) {
        launch_chained(operator_threshold_kernel, dim3((rows + 3) / 4), dim3(128), 0, st,
                       reinterpret_cast<const uint16_t*>(test_o), ve, amin, rows, H, D);
        if ((rc = cuda_status(cudaGetLastError(), "v_output threshold launch")) != AKV_OK) return rc;
    }
    rc = launch_v_compute_res(f8, m4, l4, sp, amin, takes_probe ? test_o : nullptr, ve, adds ? res : nullptr, o, B, H, 1,
                              max_seq_len, D, s_last_dim, n, reference, takes_probe, st);
    if (rc != AKV_OK || rest_len == 0 || adds) return rc;
    launch_chained(operator_add_kernel, dim3((rows * D + 255) / 256), dim3(256), 0, st, reinterpret_cast<uint16_t*>(o),
                   reinterpret_cast<const uint16_t*>(res), rows * D);
    return cuda_status(cudaGetLastError(), "v_output residual launch");
}

}  // extern "C"

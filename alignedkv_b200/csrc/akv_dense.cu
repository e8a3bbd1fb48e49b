// The element-wise parts of a decoder's decode step between its matrix products (model/Llama_AlignedKV.py's layer, as
// llama.py restates it): rotary embedding with the split into queries, keys and values, SwiGLU's activation, RMSNorm.
//   rope_split_kernel   qkv [B, H + 2 Hkv, D] -> q [B,H,D], k, v [B,Hkv,D]; q and k rotated (rotate_half form)
//   silu_mul_kernel     [rows, 2 F] (gate | up) -> silu(gate) * up
//   rms_norm_kernel     x / sqrt(mean(x^2) + eps) * w per row
// One launch each where tensor operations take 22, 2 and 1: at batch 16 every one of those is a kernel of 2 us and more that
// moves a few hundred kilobytes.  Rotation and activation are the tensor operations' bit for bit: tables and rotation in fp32,
// rounded once; silu in fp32, rounded to fp16, then an fp16 product.  The norm is computed in fp32 and rounded once, but adds its
// squares in an order of its own (about one value in 20000 is one fp16 step off torch's, which two layers turn into logits
// 8e-4 off): LlamaDecoder takes torch's, one launch as well.
#include "akv_common.cuh"

namespace akv {
namespace {

constexpr int ROPE_NT = 128;

// Thread = 8 channels of a head and the 8 half a head further; D / 16 threads per head.
__global__ void __launch_bounds__(ROPE_NT)
rope_split_kernel(const uint16_t* __restrict__ qkv, const long long* __restrict__ pos, uint16_t* __restrict__ q,
                  uint16_t* __restrict__ k, uint16_t* __restrict__ v, int H, int Hkv, int D, float theta) {
    __shared__ __align__(16) float cs[128], sn[128];
    const int hd = D >> 1, per = D >> 4, tid = threadIdx.x;
    // (the same fp32 operations as the prompt's tables, llama.py: a position is rotated alike in both)
    const float at = (float)pos[0], inv_d = 1.f / (float)D;
    for (int i = tid; i < hd; i += ROPE_NT) {
        const float a = at * (1.f / powf(theta, (float)(2 * i) * inv_d));
        cs[i] = cosf(a);
        sn[i] = sinf(a);
    }
    __syncthreads();
    const int heads = H + 2 * Hkv, b = blockIdx.x;
    const int head = blockIdx.y * (ROPE_NT / per) + tid / per, c = (tid % per) * 8;
    if (tid >= ROPE_NT / per * per || head >= heads) return;
    const uint16_t* src = qkv + ((size_t)b * heads + head) * D + c;
    uint4 lo = *reinterpret_cast<const uint4*>(src), hi = *reinterpret_cast<const uint4*>(src + hd);
    if (head < H + Hkv) {
        __half2* l2 = reinterpret_cast<__half2*>(&lo);
        __half2* h2 = reinterpret_cast<__half2*>(&hi);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float2 x = __half22float2(l2[j]), y = __half22float2(h2[j]);
            const float c0 = cs[c + 2 * j], c1 = cs[c + 2 * j + 1], s0 = sn[c + 2 * j], s1 = sn[c + 2 * j + 1];
            l2[j] = __floats2half2_rn(fmaf(y.x, -s0, x.x * c0), fmaf(y.y, -s1, x.y * c1));
            h2[j] = __floats2half2_rn(fmaf(x.x, s0, y.x * c0), fmaf(x.y, s1, y.y * c1));
        }
    }
    uint16_t* dst = head < H ? q + ((size_t)b * H + head) * D
                  : head < H + Hkv ? k + ((size_t)b * Hkv + head - H) * D : v + ((size_t)b * Hkv + head - H - Hkv) * D;
    *reinterpret_cast<uint4*>(dst + c) = lo;
    *reinterpret_cast<uint4*>(dst + c + hd) = hi;
}

__global__ void __launch_bounds__(128)
silu_mul_kernel(const uint16_t* __restrict__ gate_up, uint16_t* __restrict__ out, int F) {
    const size_t row = blockIdx.x;
    const uint16_t *gate = gate_up + row * 2 * F, *up = gate + F;
    for (int i = (blockIdx.y * 128 + threadIdx.x) * 8; i < F; i += gridDim.y * 1024) {
        const uint4 g4 = *reinterpret_cast<const uint4*>(gate + i), u4 = *reinterpret_cast<const uint4*>(up + i);
        uint4 o4;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float2 g = __half22float2(reinterpret_cast<const __half2*>(&g4)[j]);
            const __half2 a = __floats2half2_rn(g.x / (1.f + expf(-g.x)), g.y / (1.f + expf(-g.y)));
            reinterpret_cast<__half2*>(&o4)[j] = __hmul2(a, reinterpret_cast<const __half2*>(&u4)[j]);
        }
        *reinterpret_cast<uint4*>(out + row * F + i) = o4;
    }
}

// One CTA per row, its values in registers between the sum and the scaling: one pass over memory, one reduction.
constexpr int NORM_NT = 512, NORM_V = 4;      // vectors of 8 a thread holds: rows of up to 16384 values
__global__ void __launch_bounds__(NORM_NT)
rms_norm_kernel(const uint16_t* __restrict__ x, const uint16_t* __restrict__ w, uint16_t* __restrict__ out, int n, float eps) {
    __shared__ float red[NORM_NT / 32];
    const int tid = threadIdx.x, nv = n >> 3;
    const uint4* src = reinterpret_cast<const uint4*>(x + (size_t)blockIdx.x * n);
    uint4 a[NORM_V], g[NORM_V];
    float sum = 0.f;
#pragma unroll
    for (int j = 0; j < NORM_V; ++j) {
        const int v = tid + j * NORM_NT;
        if (v < nv) {
            a[j] = src[v];
            g[j] = __ldg(reinterpret_cast<const uint4*>(w) + v);
        }
    }
#pragma unroll
    for (int j = 0; j < NORM_V; ++j) {
        if (tid + j * NORM_NT >= nv) break;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 f = __half22float2(reinterpret_cast<const __half2*>(&a[j])[i]);
            sum = fmaf(f.x, f.x, sum);
            sum = fmaf(f.y, f.y, sum);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
    if ((tid & 31) == 0) red[tid >> 5] = sum;
    __syncthreads();
    sum = red[tid & (NORM_NT / 32 - 1)];
#pragma unroll
    for (int o = NORM_NT / 64; o > 0; o >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
    const float r = rsqrtf(sum / (float)n + eps);
    uint4* dst = reinterpret_cast<uint4*>(out + (size_t)blockIdx.x * n);
#pragma unroll
    for (int j = 0; j < NORM_V; ++j) {
        const int v = tid + j * NORM_NT;
        if (v >= nv) break;
        uint4 o4;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 f = __half22float2(reinterpret_cast<const __half2*>(&a[j])[i]);
            const float2 h = __half22float2(reinterpret_cast<const __half2*>(&g[j])[i]);
            reinterpret_cast<__half2*>(&o4)[i] = __floats2half2_rn(f.x * r * h.x, f.y * r * h.y);
        }
        dst[v] = o4;
    }
}

}  // namespace
}  // namespace akv

using namespace akv;

extern "C" {

int akv_rope_split(const void* qkv, const void* pos, void* q, void* k, void* v, int bsz, int n_heads, int n_kv_heads,
                   int head_dim, float theta, void* stream) {
    set_error("");
    AKV_REQUIRE(qkv && pos && q && k && v, AKV_ERR_NULL, "rope_split: null pointer");
    AKV_REQUIRE(bsz > 0 && n_heads > 0 && n_kv_heads > 0 && head_dim > 0 && head_dim % 16 == 0 && head_dim <= 256 &&
                n_heads + 2ll * n_kv_heads <= 65535, AKV_ERR_SHAPE, "rope_split: unsupported extent (bsz %d, heads %d + 2 x %d, "
                "head_dim %d [multiple of 16, at most 256])", bsz, n_heads, n_kv_heads, head_dim);
    AKV_REQUIRE(aligned16(qkv) && aligned16(q) && aligned16(k) && aligned16(v) && (reinterpret_cast<uintptr_t>(pos) & 7u) == 0,
                AKV_ERR_ALIGN, "rope_split: pointers must be 16-byte aligned");
    const int per = ROPE_NT / (head_dim >> 4);
    count_launch();
    rope_split_kernel<<<dim3(bsz, (n_heads + 2 * n_kv_heads + per - 1) / per), ROPE_NT, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const uint16_t*>(qkv), static_cast<const long long*>(pos), static_cast<uint16_t*>(q),
        static_cast<uint16_t*>(k), static_cast<uint16_t*>(v), n_heads, n_kv_heads, head_dim, theta);
    return cuda_status(cudaGetLastError(), "rope_split launch");
}

int akv_silu_mul(const void* gate_up, void* out, int rows, int width, void* stream) {
    set_error("");
    AKV_REQUIRE(gate_up && out, AKV_ERR_NULL, "silu_mul: null pointer");
    AKV_REQUIRE(rows > 0 && width > 0 && width % 8 == 0 && width <= (1 << 30), AKV_ERR_SHAPE,
                "silu_mul: unsupported extent (%d rows of %d [multiple of 8])", rows, width);
    AKV_REQUIRE(aligned16(gate_up) && aligned16(out), AKV_ERR_ALIGN, "silu_mul: pointers must be 16-byte aligned");
    count_launch();
    const int across = (width / 8 + 127) / 128;
    silu_mul_kernel<<<dim3(rows, across < 65535 ? across : 65535), 128, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const uint16_t*>(gate_up), static_cast<uint16_t*>(out), width);
    return cuda_status(cudaGetLastError(), "silu_mul launch");
}

int akv_rms_norm(const void* x, const void* w, void* out, int rows, int width, float eps, void* stream) {
    set_error("");
    AKV_REQUIRE(x && w && out, AKV_ERR_NULL, "rms_norm: null pointer");
    AKV_REQUIRE(rows > 0 && width > 0 && width % 8 == 0 && width <= 8 * NORM_V * NORM_NT, AKV_ERR_SHAPE,
                "rms_norm: unsupported extent (%d rows of %d [multiple of 8, at most %d])", rows, width, 8 * NORM_V * NORM_NT);
    AKV_REQUIRE(aligned16(x) && aligned16(w) && aligned16(out), AKV_ERR_ALIGN, "rms_norm: pointers must be 16-byte aligned");
    count_launch();
    rms_norm_kernel<<<rows, NORM_NT, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const uint16_t*>(x), static_cast<const uint16_t*>(w), static_cast<uint16_t*>(out), width, eps);
    return cuda_status(cudaGetLastError(), "rms_norm launch");
}

}  // extern "C"

// Prompt ingestion in one pass: what K_Cache_Class.save / V_Cache_Class.save do for start_pos == 0
// (extension/k_cache_file.py:76-96, extension/v_cache_file.py:79-96) - per-channel exponent of the signed maximum over
// the prompt, whole 64-token blocks split into the planes (K1 / V1: extension/csrc/K_cache.cu:19-58,
// extension/csrc/V_cache.cu:17-41), the remaining tokens copied to the fp16 residual buffers - reading every input
// byte once.  The reference makes three passes per tensor (max reduction, plane writer, tail copy).
//
// prefill128_kernel (head_dim 128): grid (ceil(S/64), H, B), 256 threads, one 64-token tile of K and of V per CTA.
// Every plane piece of a tile - a K block's three planes, 64 V rows' three planes - is contiguous in memory: the results
// are put together in shared memory, over the input tile, and leave by six bulk stores.  prefill_kernel: any other head
// size, and the same partial maxima.  exp_reduce_kernel takes the maximum over tiles and stores its exponent field.
#include "akv_save.cuh"

namespace akv {

constexpr int PF_BLK = 64;

__global__ void __launch_bounds__(128)
prefill_kernel(uint8_t* __restrict__ k_first_8, uint8_t* __restrict__ k_mid_4, uint8_t* __restrict__ k_last_4,
               uint8_t* __restrict__ v_first_8, uint8_t* __restrict__ v_mid_4, uint8_t* __restrict__ v_last_4,
               uint8_t* __restrict__ restk, uint8_t* __restrict__ restv, const uint8_t* __restrict__ k,
               const uint8_t* __restrict__ v, uint16_t* __restrict__ kmax_part, uint16_t* __restrict__ vmax_part, int H,
               int D, int S, int nmb, int max_seq_len, int tiles) {
    extern __shared__ __align__(16) uint8_t smem[];      // K tile, then V tile: [64][D] halves each
    const int z = blockIdx.x, h = blockIdx.y;
    const long long b = blockIdx.z;
    const long long bh = b * H + h;
    const int t0 = z * PF_BLK;
    const int cnt = min(PF_BLK, S - t0);
    const int pitch = 2 * D;
    uint8_t* ks = smem;
    uint8_t* vs = smem + PF_BLK * pitch;
    auto krow = [&](int t) { return k + 2 * (((b * S + t0 + t) * H + h) * (long long)D); };
    auto vrow = [&](int t) { return v + 2 * (((b * S + t0 + t) * H + h) * (long long)D); };
    stage_tile64(ks, krow, D, cnt);
    stage_tile64(vs, vrow, D, cnt);
    __syncthreads();
    uint16_t* kmx = kmax_part + (bh * tiles + z) * D;
    uint16_t* vmx = vmax_part + (bh * tiles + z) * D;
    if (cnt == PF_BLK) {
        k_emit_block64<true>(ks, k_first_8, k_mid_4, k_last_4, bh * nmb + z, D, kmx);
        // V rows: 64 tokens x D/32 pieces
        const int per_tok = D >> 5;
        for (int i = threadIdx.x; i < PF_BLK * per_tok; i += blockDim.x) {
            const int t = i / per_tok, c = i - t * per_tok;
            const size_t prow = (size_t)bh * max_seq_len + t0 + t;
            const uint4* src = reinterpret_cast<const uint4*>(vs + t * pitch + c * 64);      // shared memory
            v_write32(src[0], src[1], src[2], src[3], v_first_8 + prow * D + c * 32, v_mid_4 + prow * (D >> 1) + c * 16,
                      v_last_4 + prow * (D >> 1) + c * 16);
        }
    } else {
        // the prompt's last, partial tile stays in fp16 (residual buffers [B,64,H,D], rows 0..cnt-1)
        const int vec_per_row = pitch >> 4;
        for (int i = threadIdx.x; i < cnt * vec_per_row; i += blockDim.x) {
            const int t = i / vec_per_row, vv = i - t * vec_per_row;
            const size_t dst = 2 * ((((size_t)b * PF_BLK + t) * H + h) * (size_t)D) + vv * 16;
            *reinterpret_cast<uint4*>(restk + dst) = *reinterpret_cast<const uint4*>(ks + t * pitch + vv * 16);
            *reinterpret_cast<uint4*>(restv + dst) = *reinterpret_cast<const uint4*>(vs + t * pitch + vv * 16);
        }
    }
    // per-channel signed maxima of the tile (K's come out of the block writer when the tile is whole)
    for (int d = threadIdx.x; d < D; d += blockDim.x) {
        float vm = -INFINITY, km = -INFINITY;
        for (int t = 0; t < cnt; ++t) {
            vm = fmaxf(vm, __half2float(*reinterpret_cast<const __half*>(vs + t * pitch + 2 * d)));
            if (cnt != PF_BLK) km = fmaxf(km, __half2float(*reinterpret_cast<const __half*>(ks + t * pitch + 2 * d)));
        }
        vmx[d] = __half_as_ushort(__float2half_rn(vm));
        if (cnt != PF_BLK) kmx[d] = __half_as_ushort(__float2half_rn(km));
    }
}

// ---- head_dim 128
namespace pf {
constexpr int D = 128, NT = 256, IN_BYTES = PF_BLK * 2 * D;          // one tile as it arrives
// Row t of a staged tile: 256 bytes, 32 bytes further after every 16 tokens - four threads that read the same channels of
// tokens 16 apart then hit different banks.
constexpr int BUF_BYTES = IN_BYTES + 128;
__device__ __forceinline__ int row_at(int t) { return t * 2 * D + (t >> 4) * 32; }
}  // namespace pf

__device__ __forceinline__ uint32_t hmax2_bits(uint32_t a, uint32_t b) {
    const __half2 r = __hmax2(*reinterpret_cast<const __half2*>(&a), *reinterpret_cast<const __half2*>(&b));
    return *reinterpret_cast<const uint32_t*>(&r);
}
__device__ __forceinline__ void bulk_store(void* dst, uint32_t src, uint32_t bytes) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;\n" ::"l"(dst), "r"(src), "r"(bytes) : "memory");
}
// Four tokens' low bytes of a channel [t0, t1, t2, t3] -> two bytes of a nibble plane (in bytes 0 and 2), the even token's
// nibble above the odd one's (extension/csrc/K_cache.cu:49-56)
__device__ __forceinline__ uint32_t mid_nibbles(uint32_t x) { return (x & 0x00F000F0u) | ((x >> 12) & 0x000F000Fu); }
__device__ __forceinline__ uint32_t low_nibbles(uint32_t x) { return ((x << 4) & 0x00F000F0u) | ((x >> 8) & 0x000F000Fu); }

// ADD: the K nibbles are added onto what the planes hold, as the reference's writer does (DecodeLayer.prefill); else they are
// stored, for a caller of the library that knows the planes to be zero there: batch 8 x 32 heads x 4096 tokens 200.7 us with the
// rewind, 219.5 with ADD.  A layer cannot know: a tensor's version counter sees no writer that has its address (this library's
// K block writer, `.data`, DLPack).  (Launched with programmatic serialization it took 228, and the maxima so launched 270.)
// Bound by HBM: 32 KB in, 32 KB out and, with ADD, 8 KB of nibble planes read per tile.  Thread = (channel pair c = tid / 4, 16
// tokens q = tid % 4): 16 four-byte shared loads of a tile give 2 x (16 high bytes, 8 mid, 8 low bytes) of the K planes, all
// transposition by byte permutes; for V = (token, 32 channels).  About 4 integer instructions per value where the form before it
// (thread = channel, one 2-byte load per value, results stored 16 bytes at a time straight to the planes) took 10 and half-filled
// every sector it wrote: batch 8 x 32 heads x 4096 tokens 182.5 us with ADD (1.21 GB: 6.6 TB/s) against 356.4.
template <bool ADD>
__global__ void __launch_bounds__(pf::NT, 4)
prefill128_kernel(uint8_t* __restrict__ k_first_8, uint8_t* __restrict__ k_mid_4, uint8_t* __restrict__ k_last_4,
                  uint8_t* __restrict__ v_first_8, uint8_t* __restrict__ v_mid_4, uint8_t* __restrict__ v_last_4,
                  uint8_t* __restrict__ restk, uint8_t* __restrict__ restv, const uint8_t* __restrict__ k,
                  const uint8_t* __restrict__ v, uint32_t* __restrict__ kmax_part, uint32_t* __restrict__ vmax_part, int H,
                  int S, int nmb, int max_seq_len, int tiles) {
    using namespace pf;
    __shared__ __align__(128) uint8_t ks[BUF_BYTES], vs[BUF_BYTES];
    const int tid = threadIdx.x, z = blockIdx.x, h = blockIdx.y;
    const long long b = blockIdx.z, bh = b * H + h;
    const int t0 = z * PF_BLK, cnt = min(PF_BLK, S - t0);
    const size_t in0 = ((size_t)(b * S + t0) * H + h) * (2 * D), in_step = (size_t)H * 2 * D;
    const uint32_t ka = smem_u32(ks), va = smem_u32(vs);
#pragma unroll
    for (int j = 0; j < IN_BYTES / 16 / NT; ++j) {
        const int i = tid + j * NT, t = i >> 4, o = (i & 15) * 16;
        if (t < cnt) {
            cp_async16(ka + row_at(t) + o, k + in0 + t * in_step + o);
            cp_async16(va + row_at(t) + o, v + in0 + t * in_step + o);
        }
    }
    cp_async_commit();
    const int c = tid >> 2, q = tid & 3;                             // channel pair, tokens 16 q .. 16 q + 15
    const size_t tile = (size_t)(bh * nmb + z) * D;                  // plane row of channel 0
    uint8_t* mid = k_mid_4 + (tile + 2 * c) * 32 + q * 8;
    uint8_t* low = k_last_4 + (tile + 2 * c) * 32 + q * 8;
    uint2 om[2], ol[2];                                              // the nibble bytes this thread adds onto
    if (ADD && cnt == PF_BLK) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            om[e] = *reinterpret_cast<const uint2*>(mid + e * 32);
            ol[e] = *reinterpret_cast<const uint2*>(low + e * 32);
        }
    }
    cp_async_wait<0>();
    __syncthreads();
    // signed maxima of this thread's channel pair over its tokens (extension/k_cache_file.py:77-78), as fp16x2
    uint32_t km = 0xFC00FC00u, vm = 0xFC00FC00u;
    uint32_t kw[16];
#pragma unroll
    for (int t = 0; t < 16; ++t) {
        const int a = row_at(16 * q + t) + 4 * c;
        kw[t] = *reinterpret_cast<const uint32_t*>(ks + a);
        const uint32_t vw = *reinterpret_cast<const uint32_t*>(vs + a);
        if (16 * q + t < cnt) {
            km = hmax2_bits(km, kw[t]);
            vm = hmax2_bits(vm, vw);
        }
    }
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) {
        km = hmax2_bits(km, __shfl_xor_sync(0xFFFFFFFFu, km, o));
        vm = hmax2_bits(vm, __shfl_xor_sync(0xFFFFFFFFu, vm, o));
    }
    if (q == 0) {
        const size_t at = (size_t)(bh * tiles + z) * (D / 2) + c;
        kmax_part[at] = km;
        vmax_part[at] = vm;
    }
    if (cnt < PF_BLK) {
        // the prompt's last, partial tile stays in fp16 (residual buffers [B,64,H,D], rows 0..cnt-1)
        for (int i = tid; i < cnt * 16; i += NT) {
            const int t = i >> 4, o = (i & 15) * 16;
            const size_t dst = ((size_t)(b * PF_BLK + t) * H + h) * (2 * D) + o;
            *reinterpret_cast<uint4*>(restk + dst) = *reinterpret_cast<const uint4*>(ks + row_at(t) + o);
            *reinterpret_cast<uint4*>(restv + dst) = *reinterpret_cast<const uint4*>(vs + row_at(t) + o);
        }
        return;
    }
    // K: per 4 tokens, words [lo a, hi a, lo b, hi b] of channels a, b -> high bytes and low bytes of each channel
    uint32_t f[2][4], m[2][2], l[2][2];
#pragma unroll
    for (int g = 0; g < 2; ++g) {                                    // 8 tokens
        uint32_t lo[2][2];
#pragma unroll
        for (int p = 0; p < 2; ++p) {                                // 4 tokens
            const uint32_t* w = kw + 8 * g + 4 * p;
            const uint32_t h01 = __byte_perm(w[0], w[1], 0x7531), h23 = __byte_perm(w[2], w[3], 0x7531);
            const uint32_t l01 = __byte_perm(w[0], w[1], 0x6420), l23 = __byte_perm(w[2], w[3], 0x6420);
            f[0][2 * g + p] = __byte_perm(h01, h23, 0x6420);
            f[1][2 * g + p] = __byte_perm(h01, h23, 0x7531);
            lo[0][p] = __byte_perm(l01, l23, 0x6420);
            lo[1][p] = __byte_perm(l01, l23, 0x7531);
        }
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            m[e][g] = __byte_perm(mid_nibbles(lo[e][0]), mid_nibbles(lo[e][1]), 0x6420);
            l[e][g] = __byte_perm(low_nibbles(lo[e][0]), low_nibbles(lo[e][1]), 0x6420);
        }
    }
#pragma unroll
    for (int e = 0; ADD && e < 2; ++e) {                             // bytewise, modulo 256
        m[e][0] = __vadd4(m[e][0], om[e].x);
        m[e][1] = __vadd4(m[e][1], om[e].y);
        l[e][0] = __vadd4(l[e][0], ol[e].x);
        l[e][1] = __vadd4(l[e][1], ol[e].y);
    }
    // V: token t, 32 channels
    const int t = tid >> 2;
    uint4 vf0, vf1, vmid, vlow;
    {
        const uint4* src = reinterpret_cast<const uint4*>(vs + row_at(t) + q * 64);
        const uint4 a0 = src[0], a1 = src[1], a2 = src[2], a3 = src[3];
        v_split4(a0.x, a0.y, a0.z, a0.w, vf0.x, vf0.y, vmid.x, vlow.x);
        v_split4(a1.x, a1.y, a1.z, a1.w, vf0.z, vf0.w, vmid.y, vlow.y);
        v_split4(a2.x, a2.y, a2.z, a2.w, vf1.x, vf1.y, vmid.z, vlow.z);
        v_split4(a3.x, a3.y, a3.z, a3.w, vf1.z, vf1.w, vmid.w, vlow.w);
    }
    __syncthreads();                                                 // (the tiles have been read)
    // planes in the order of memory: high [0, 8 KB), mid, low (4 KB each).  Threads next to each other write different
    // halves of a row first, so that a warp's stores spread over the banks.
#pragma unroll
    for (int s = 0; s < 2; ++s) {
        const int e = s ^ (c & 1), n = s ^ ((c >> 1) & 1);
        const uint32_t x = e ? f[1][0] : f[0][0], y = e ? f[1][1] : f[0][1], zz = e ? f[1][2] : f[0][2], w = e ? f[1][3] : f[0][3];
        *reinterpret_cast<uint4*>(ks + (2 * c + e) * 64 + q * 16) = make_uint4(x, y, zz, w);
        *reinterpret_cast<uint2*>(ks + 8192 + (2 * c + n) * 32 + q * 8) = n ? make_uint2(m[1][0], m[1][1]) : make_uint2(m[0][0], m[0][1]);
        *reinterpret_cast<uint2*>(ks + 12288 + (2 * c + n) * 32 + q * 8) = n ? make_uint2(l[1][0], l[1][1]) : make_uint2(l[0][0], l[0][1]);
    }
    *reinterpret_cast<uint4*>(vs + t * 128 + q * 32) = vf0;
    *reinterpret_cast<uint4*>(vs + t * 128 + q * 32 + 16) = vf1;
    *reinterpret_cast<uint4*>(vs + 8192 + t * 64 + q * 16) = vmid;
    *reinterpret_cast<uint4*>(vs + 12288 + t * 64 + q * 16) = vlow;
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    __syncthreads();
    if (tid == 0) {
        const size_t vrow = (size_t)bh * max_seq_len + t0;
        bulk_store(k_first_8 + tile * 64, ka, 8192);
        bulk_store(k_mid_4 + tile * 32, ka + 8192, 4096);
        bulk_store(k_last_4 + tile * 32, ka + 12288, 4096);
        bulk_store(v_first_8 + vrow * D, va, 8192);
        bulk_store(v_mid_4 + vrow * (D / 2), va + 8192, 4096);
        bulk_store(v_last_4 + vrow * (D / 2), va + 12288, 4096);
        asm volatile("cp.async.bulk.commit_group;\n" ::: "memory");
        asm volatile("cp.async.bulk.wait_group 0;\n" ::: "memory");  // (shared memory is read, and the planes are written)
    }
}

// exponent field of the signed maximum over the tiles -> [B,1,H,D] bytes.  Thread = (channel pair, share of the tiles).
__global__ void __launch_bounds__(256)
exp_reduce_kernel(const uint32_t* __restrict__ kmax_part, const uint32_t* __restrict__ vmax_part,
                  uint8_t* __restrict__ k_exp, uint8_t* __restrict__ v_exp, int hd, int tiles) {
    __shared__ uint32_t red[2][256];
    const long long bh = blockIdx.x;
    const int shares = hd <= 128 ? 256 / hd : 1;                     // (hd <= 128: head_dim is at most 256)
    const int c = threadIdx.x % hd, g = threadIdx.x / hd;
    uint32_t km = 0xFC00FC00u, vm = 0xFC00FC00u;
    if (g < shares) {
        const size_t at = (size_t)bh * tiles * hd + c;
#pragma unroll 8
        for (int z = g; z < tiles; z += shares) {
            km = hmax2_bits(km, kmax_part[at + (size_t)z * hd]);
            vm = hmax2_bits(vm, vmax_part[at + (size_t)z * hd]);
        }
    }
    red[0][threadIdx.x] = km;
    red[1][threadIdx.x] = vm;
    __syncthreads();
    if (g == 0) {
        for (int s = 1; s < shares; ++s) {
            km = hmax2_bits(km, red[0][c + s * hd]);
            vm = hmax2_bits(vm, red[1][c + s * hd]);
        }
        const size_t at = 2 * ((size_t)bh * hd + c);                 // (the exponent tensors may lie at any address)
        k_exp[at] = (uint8_t)((km >> 10) & 0x1Fu);
        k_exp[at + 1] = (uint8_t)((km >> 26) & 0x1Fu);
        v_exp[at] = (uint8_t)((vm >> 10) & 0x1Fu);
        v_exp[at + 1] = (uint8_t)((vm >> 26) & 0x1Fu);
    }
}

}  // namespace akv

using namespace akv;

extern "C" {

long long akv_prefill_scratch_bytes(int bsz, int n_kv_heads, int head_dim, int seqlen) {
    if (bsz <= 0 || n_kv_heads <= 0 || head_dim <= 0 || seqlen <= 0) return -1;
    const long long tiles = (seqlen + PF_BLK - 1) / PF_BLK;
    return 2ll * bsz * n_kv_heads * tiles * head_dim * 2;
}

int akv_prefill_ex(void* k_first_8, void* k_mid_4, void* k_last_4, void* v_first_8, void* v_mid_4, void* v_last_4,
                   void* k_exp_max, void* v_exp_max, void* restk, void* restv, const void* k, const void* v,
                   void* scratch, long long scratch_bytes, int bsz, int n_kv_heads, int head_dim, int max_seq_len,
                   int seqlen, int flags, void* stream) {
    set_error("");
    const int B = bsz, H = n_kv_heads, D = head_dim, S = seqlen;
    AKV_REQUIRE(k_first_8 && k_mid_4 && k_last_4 && v_first_8 && v_mid_4 && v_last_4 && k_exp_max && v_exp_max &&
                restk && restv && k && v && scratch, AKV_ERR_NULL, "prefill: null pointer");
    AKV_REQUIRE(B > 0 && B <= 65535 && H > 0 && H <= 65535 && D > 0 && D % 32 == 0 && D <= 256 && S > 0 &&
                S <= max_seq_len, AKV_ERR_SHAPE, "prefill: unsupported extent (bsz %d, heads %d, head_dim %d [multiple "
                "of 32, at most 256], seqlen %d, max_seq_len %d)", B, H, D, S, max_seq_len);
    AKV_REQUIRE((flags & ~AKV_PREFILL_STORE) == 0, AKV_ERR_SHAPE, "prefill: unknown flags %d", flags);
    AKV_REQUIRE(scratch_bytes >= akv_prefill_scratch_bytes(B, H, D, S), AKV_ERR_SHAPE,
                "prefill: scratch of %lld bytes is too small", scratch_bytes);
    AKV_REQUIRE(aligned16(k_first_8) && aligned16(k_mid_4) && aligned16(k_last_4) && aligned16(v_first_8) &&
                aligned16(v_mid_4) && aligned16(v_last_4) && aligned16(restk) && aligned16(restv) && aligned16(k) &&
                aligned16(v) && aligned16(scratch), AKV_ERR_ALIGN, "prefill: pointers must be 16-byte aligned");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int tiles = (S + PF_BLK - 1) / PF_BLK;
    const int nmb = (max_seq_len + PF_BLK - 1) / PF_BLK;
    uint16_t* kmax_part = static_cast<uint16_t*>(scratch);
    uint16_t* vmax_part = kmax_part + (size_t)B * H * tiles * D;
    dim3 grid(tiles, H, B);
    count_launch(2);
    if (D == pf::D) {
        const auto kern = (flags & AKV_PREFILL_STORE) ? prefill128_kernel<false> : prefill128_kernel<true>;
        kern<<<grid, pf::NT, 0, st>>>(
            static_cast<uint8_t*>(k_first_8), static_cast<uint8_t*>(k_mid_4), static_cast<uint8_t*>(k_last_4),
            static_cast<uint8_t*>(v_first_8), static_cast<uint8_t*>(v_mid_4), static_cast<uint8_t*>(v_last_4),
            static_cast<uint8_t*>(restk), static_cast<uint8_t*>(restv), static_cast<const uint8_t*>(k),
            static_cast<const uint8_t*>(v), reinterpret_cast<uint32_t*>(kmax_part), reinterpret_cast<uint32_t*>(vmax_part), H,
            S, nmb, max_seq_len, tiles);
    } else {
        const size_t smem = (size_t)2 * PF_BLK * 2 * D;
        if (smem > 48 * 1024) {      // (the device's maximum, not this call's size: the attribute is shared by all host threads)
            cudaError_t e = cudaFuncSetAttribute(prefill_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, max_dyn_smem());
            if (e != cudaSuccess) return cuda_status(e, "prefill smem attribute");
        }
        prefill_kernel<<<grid, 128, smem, st>>>(
            static_cast<uint8_t*>(k_first_8), static_cast<uint8_t*>(k_mid_4), static_cast<uint8_t*>(k_last_4),
            static_cast<uint8_t*>(v_first_8), static_cast<uint8_t*>(v_mid_4), static_cast<uint8_t*>(v_last_4),
            static_cast<uint8_t*>(restk), static_cast<uint8_t*>(restv), static_cast<const uint8_t*>(k),
            static_cast<const uint8_t*>(v), kmax_part, vmax_part, H, D, S, nmb, max_seq_len, tiles);
    }
    int rc = cuda_status(cudaGetLastError(), "prefill launch");
    if (rc != AKV_OK) return rc;
    exp_reduce_kernel<<<B * H, 256, 0, st>>>(reinterpret_cast<const uint32_t*>(kmax_part), reinterpret_cast<const uint32_t*>(vmax_part),
                                            static_cast<uint8_t*>(k_exp_max), static_cast<uint8_t*>(v_exp_max), D / 2, tiles);
    return cuda_status(cudaGetLastError(), "prefill reduce launch");
}

int akv_prefill(void* k_first_8, void* k_mid_4, void* k_last_4, void* v_first_8, void* v_mid_4, void* v_last_4,
                void* k_exp_max, void* v_exp_max, void* restk, void* restv, const void* k, const void* v,
                void* scratch, long long scratch_bytes, int bsz, int n_kv_heads, int head_dim, int max_seq_len,
                int seqlen, void* stream) {
    return akv_prefill_ex(k_first_8, k_mid_4, k_last_4, v_first_8, v_mid_4, v_last_4, k_exp_max, v_exp_max, restk, restv, k, v,
                          scratch, scratch_bytes, bsz, n_kv_heads, head_dim, max_seq_len, seqlen, 0, stream);
}

}  // extern "C"

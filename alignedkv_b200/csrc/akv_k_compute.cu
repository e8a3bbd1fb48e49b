// Precision-aligned q.K^T over the quantized K blocks.
//
// Replaces the reference's k_cache_compute_kernel (extension/csrc/K_cache.cu:174-310).  Results are
// bit-identical: every token's score is the fp16 fused-multiply-add chain over channels 0..D-1 followed by one
// fp16 multiply with half(sqrt_dim), and a nibble plane that the alignment rule skips is replaced by the same
// constants (K_cache.cu:201-205,249-252).
//
// Design (B200): the kernel is a pure HBM stream.  Each WARP owns a private ring of shared-memory stages that
// it fills with 16-byte asynchronous copies and drains itself - no block-level barrier exists.  A warp works
// through a contiguous run of units; a unit is 4 consecutive 64-token blocks of one (batch, KV head), or one block (few blocks
// and groups of four or eight, see the launcher), and a stage holds KCH channels of the unit's blocks: the high-byte rows plus,
// only for the channels whose alignment code asks for them, the 32-byte rows of the mid / low nibble planes (rows that are
// skipped are never requested from memory).  With four blocks lane (tile, i) owns tokens 8i..8i+7 of its tile and keeps four
// fp16x2 accumulators per query head: one 8-byte and two 4-byte shared loads feed four FMAs; with one block it owns tokens
// 2i, 2i+1 and one accumulator.  No cross-lane reduction exists, which is what keeps the channel-order fp16 sum exact.
// Grouped-query attention (G query heads per KV head): a row is fetched when ANY head of the group needs it, every
// staged row is read from shared memory once and applied to the G heads in turn, each head substituting the
// reference's constants where its own code skips the plane - so plane bytes cross HBM once per group and the
// results equal G independent multi-head passes.  A row's four fp16x2 words are assembled once, with all planes; a head's
// words are (word & mask) | constant, mask and constant by the head's code on the channel: ONE logic operation per FMA (whatever
// lies in a plane's slot that the union did not fetch is masked away).  Mask, constant and query of a (head, channel) are
// tabulated when the (batch, KV head) starts.  Per row of four 64-token tiles that is 24 operations on the half-rate
// integer pipe and 16 FMAs for four heads; parking the low bytes of each code in shared memory and fetching them back per
// head, which this replaces, took 80 instructions: groups of eight 253 against
// 177 us at batch 64 x 4 KV heads x 8192 tokens, of two 56 against 46 at batch 16 x 16 x 4096, of four 41.5 against 35.5 at
// batch 8 x 8 x 8192 but 228 against 223 at batch 64 (198 since the head size is known at compile time, see the kernel), where the
// copies are what is left (a stage's issue stalls for 450 to 770 cycles on the load unit; neither bulk copies nor TMA boxes, built
// and bit-exact, moved these pieces faster).
// With G == 1 the producer writes the constants into the skipped rows' slots instead.
// In a decode step that flushes no block the kernel makes its alignment inputs itself and runs beside the append kernel in front of
// it (KParams::k_exp): batch 8 x 32 heads x 4096 tokens 80.5 -> 78.7 us per step, 16 x 32 x 1000 56.6 -> 53.0, one sequence of
// 16384 tokens 54.4 -> 53.3.  Bulk copies of the pieces (high bytes and mid plane, 1 KB and 512 bytes) were built again for this
// form and are slower: 80.3, 54.0, and 8 KV heads x 4, batch 64 x 8192 tokens 532 against 512.
#include <atomic>
#include <type_traits>

#include "akv_common.cuh"

namespace akv {

namespace kc {
constexpr int MAX_D = 256;
// A unit = TILES consecutive 64-token blocks, a stage = KCH channels of them.  (Padding: the tiles of a stage lie on distinct banks.)
__host__ __device__ constexpr int f_tile(int kch, int tiles) { return kch * 64 + (tiles > 1 ? 64 : 0); }
__host__ __device__ constexpr int n_tile(int kch, int tiles) { return kch * 32 + (tiles > 1 ? 32 : 0); }
__host__ __device__ constexpr int stage_bytes(int kch, int tiles) { return tiles * (f_tile(kch, tiles) + 2 * n_tile(kch, tiles)); }
// Per warp: two sets of union masks (16 words) and the consumer's tables.  Two sets are enough while the producer, STAGES - 1
// stages ahead, is at most one (batch, KV head) ahead: the launcher takes no ring of more stages than a unit has (with five
// stages of 16 channels and D = 64 it issued the last stage of the next head, and loaded the set after that over the current
// one, before the current head's last stage was multiplied).  G == 1: D words q (both halves equal), two
// sets that come and go with the masks.  G > 1, one set, loaded when the consumer enters a (batch, KV head): per query head
// D words mask and D words constant (of the head's alignment code on the channel), D fp16 q.
constexpr int MASK_BYTES = 64;
__host__ __device__ constexpr int head_meta(int D, int G) { return G > 1 ? 10 * D : 4 * D; }
__host__ __device__ constexpr int meta_bytes(int D, int G) { return 2 * MASK_BYTES + (G > 1 ? G : 2) * head_meta(D, G); }
// Channels per stage and ring depth with grouped queries, warps a CTA is compiled for.  Three stages of 16 channels; groups of
// eight, whose tables are large, four of 8 (for them 177 us against 226 at batch 64 x 4 KV heads x 8 x 8192 tokens; groups
// of two 46 against 51 at batch 16 x 16 x 4096, groups of four alike at batch 64 and 35.5 against 38.6 at batch 8).
__host__ __device__ constexpr int gqa_kch(int G) { return G == 8 ? 8 : 16; }
__host__ __device__ constexpr int gqa_stages(int G) { return G == 8 ? 4 : 3; }
__host__ __device__ constexpr int max_warps(int G) { return G == 1 ? 16 : 8; }
}  // namespace kc

struct KParams {
    const uint8_t* first8;
    const uint8_t* mid4;
    const uint8_t* last4;
    const uint8_t* kq;
    const uint8_t* kqmax;
    const uint8_t* q;
    uint8_t* s;
    int BH, nb, nmb, D, ngroups;   // BH = batch x KV heads
    int units, upw;       // total units, units per warp (contiguous run)
    uint32_t scale2;      // half(sqrt_dim) in both halves
    int reference;
    // k_exp != nullptr: kq and kqmax are made here from q, the exponent maxima and the new token (k_new, null: none), which the
    // kernel in front of this one may still be storing, and the planes are read before that kernel has completed (pdl_turn)
    const uint8_t* k_exp;
    const uint16_t* k_new;
};

__device__ __forceinline__ void st_shared_v4(uint32_t a, uint32_t v) {
    asm volatile("st.shared.v4.u32 [%0], {%1,%1,%1,%1};\n" ::"r"(a), "r"(v) : "memory");
}

// Both halves of the result = half `hi` of w, and the fp16x2 multiply-add with it (the selection is part of the instruction).
__device__ __forceinline__ __half2 kc_dup(uint32_t w, int hi) {
    const __half2 h = *reinterpret_cast<const __half2*>(&w);
    return hi ? __high2half2(h) : __low2half2(h);
}
__device__ __forceinline__ uint32_t kc_fma(uint32_t k, __half2 q, uint32_t acc) {
    const __half2 r = __hfma2(*reinterpret_cast<const __half2*>(&k), q, *reinterpret_cast<const __half2*>(&acc));
    return *reinterpret_cast<const uint32_t*>(&r);
}
// A row of a stage as fp16x2 words, all planes: tokens (0, 2), (1, 3), (4, 6), (5, 7) of the lane's eight - with one tile its two.
template <int TILES>
__device__ __forceinline__ void kc_row(uint32_t (&w)[TILES], const uint8_t* f, const uint8_t* m, const uint8_t* l) {
    if (TILES == 4) {
        const uint2 fw = *reinterpret_cast<const uint2*>(f);
        const uint32_t M = *reinterpret_cast<const uint32_t*>(m), L = *reinterpret_cast<const uint32_t*>(l);
        const uint32_t lbe = (M & 0xF0F0F0F0u) | ((L >> 4) & 0x0F0F0F0Fu);   // low bytes, tokens 0,2,4,6
        const uint32_t lbo = ((M << 4) & 0xF0F0F0F0u) | (L & 0x0F0F0F0Fu);   // low bytes, tokens 1,3,5,7
        w[0] = __byte_perm(lbe, fw.x, 0x6140);
        w[1 % TILES] = __byte_perm(lbo, fw.x, 0x7150);
        w[2 % TILES] = __byte_perm(lbe, fw.y, 0x6342);
        w[3 % TILES] = __byte_perm(lbo, fw.y, 0x7352);
    } else {
        const uint32_t fw = *reinterpret_cast<const uint16_t*>(f), M = *m * 0x1001u, L = *l * 0x1001u;
        w[0] = __byte_perm((M & 0xF0F0u) | ((L >> 4) & 0x0F0Fu), fw, 0x5140);
    }
}

// Position of a stream of stages (unit, channel chunk) inside one warp's run of units.
struct KCursor {
    int u, g, bh, c;          // absolute unit, block group inside (batch, KV head), (batch, KV head), channel chunk
    int slot;                 // set of union masks of the current (batch, KV head)
    size_t row;               // plane row index of (tile 0 of the unit, first channel of the chunk)
};

// Query bits and alignment differences of heads g0 .. g0 + HC - 1 of a group on channels r * 32 + lane: mid plane read iff
// (u8)(kqmax - kq[d]) < 8, low plane iff < 4 (K_cache.cu:211,249-250).  kq and kqmax as they are given, or made here from the
// query, the exponent maxima and the new token (k_cache_file.py:98-99,136-138).
// NR: rows of 32 channels, D = 32 NR or less.  All loads go out before the first use: a warp that has two or three units pays this
// latency twice per (batch, KV head), in the masks and in the tables (19 sequences x 8 KV heads x 4 x 3968 tokens 137 us per step with
// loads a head at a time, 143 with ordered loads in functions of their own, 129 so; 8 x 4 x 8 x 10432 146.5, 149, 129).
template <int G, int HC, int NR>
__device__ __forceinline__ void kc_load_heads(const KParams& p, long long bh, int g0, int lane, uint32_t (&qh)[HC][NR],
                                              uint32_t (&diff)[HC][NR]) {
    uint32_t ek[NR], kn[NR], top[HC];
    const bool own = p.k_exp != nullptr;
#pragma unroll
    for (int r = 0; r < NR; ++r) {
        const int d = r * 32 + lane;
        const bool in = d < p.D;
        ek[r] = own && in ? ld_relaxed8(p.k_exp + bh * p.D + d) : 0u;
        kn[r] = own && p.k_new && in ? ld_relaxed16(p.k_new + bh * p.D + d) : 0u;
#pragma unroll
        for (int g = 0; g < HC; ++g) {
            const long long at = (bh * G + g0 + g) * p.D + d;
            qh[g][r] = in ? ld_relaxed16(reinterpret_cast<const uint16_t*>(p.q) + at) : 0u;
            diff[g][r] = !own && in ? __ldg(p.kq + at) : 0u;
        }
    }
#pragma unroll
    for (int g = 0; g < HC; ++g) top[g] = own ? 0u : __ldg(p.kqmax + bh * G + g0 + g);
    if (own) {
        // (old or new maximum: the token's exponent is taken in again)
#pragma unroll
        for (int r = 0; r < NR; ++r) ek[r] = max(ek[r], (kn[r] >> 10) & 0x1Fu);
#pragma unroll
        for (int g = 0; g < HC; ++g) {
#pragma unroll
            for (int r = 0; r < NR; ++r)
                if (r * 32 + lane < p.D) {
                    diff[g][r] = (((qh[g][r] >> 10) & 0x1Fu) + ek[r]) & 0xFFu;
                    top[g] = max(top[g], diff[g][r]);
                }
            top[g] = __reduce_max_sync(0xFFFFFFFFu, top[g]);
        }
    }
#pragma unroll
    for (int g = 0; g < HC; ++g)
#pragma unroll
        for (int r = 0; r < NR; ++r) diff[g][r] = p.reference ? 0u : (top[g] - diff[g][r]) & 0xFFu;
}
// The union of the group's plane-read masks (bit d set = row d of that plane is read), which is what the producer fetches; with
// one head its table too.
template <int G, int NR>
__device__ __forceinline__ void kc_load_masks(const KParams& p, long long bh, uint32_t* um, uint32_t* table, int lane) {
    constexpr int HC = G > 4 ? 4 : G;             // (registers)
    uint32_t least[NR];
#pragma unroll
    for (int r = 0; r < NR; ++r) least[r] = 0xFFu;
#pragma unroll 1
    for (int g0 = 0; g0 < G; g0 += HC) {
        uint32_t qh[HC][NR], diff[HC][NR];
        kc_load_heads<G, HC, NR>(p, bh, g0, lane, qh, diff);
#pragma unroll
        for (int r = 0; r < NR; ++r) {
            const int d = r * 32 + lane;
            if (d >= p.D) break;
#pragma unroll
            for (int g = 0; g < HC; ++g) least[r] = min(least[r], diff[g][r]);
            if (G == 1) table[d] = qh[0][r] | (qh[0][r] << 16);
        }
    }
#pragma unroll
    for (int r = 0; r < NR; ++r) {
        if (r * 32 >= p.D) break;
        const uint32_t m = __ballot_sync(0xFFFFFFFFu, least[r] < 8), l = __ballot_sync(0xFFFFFFFFu, least[r] < 4);
        if (lane == 0) {
            um[r] = m;
            um[8 + r] = l;
        }
    }
    __syncwarp();
}
// The consumer's tables of a group (all its lanes are done with the previous ones).
template <int G, int NR>
__device__ __forceinline__ void kc_load_tables(const KParams& p, long long bh, uint8_t* tables, int lane) {
    constexpr int HC = G > 4 ? 4 : G;
    __syncwarp();
#pragma unroll 1
    for (int g0 = 0; g0 < G; g0 += HC) {
        uint32_t qh[HC][NR], diff[HC][NR];
        kc_load_heads<G, HC, NR>(p, bh, g0, lane, qh, diff);
#pragma unroll
        for (int g = 0; g < HC; ++g) {
            uint32_t* hm = reinterpret_cast<uint32_t*>(tables + (size_t)(g0 + g) * kc::head_meta(p.D, G));
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                const int d = r * 32 + lane;
                if (d >= p.D) break;
                const uint32_t x = diff[g][r];
                hm[d] = x < 4 ? 0xFFFFFFFFu : x < 8 ? 0xFFF0FFF0u : 0xFF00FF00u;
                hm[p.D + d] = x < 4 ? 0u : x < 8 ? 0x00080008u : 0x00800080u;
                reinterpret_cast<uint16_t*>(hm + 2 * p.D)[d] = (uint16_t)qh[g][r];
            }
        }
    }
    __syncwarp();
}

// DC: the head size when it is known, 0 for any: the copies' addresses are then immediate offsets from two pointers, and a unit whose
// tiles all exist checks none of them.  A row of four heads took 68 instructions where the arithmetic needs 46: 8 KV heads x 4, batch
// 64 x 8192 tokens 505 -> 479 us per step, 8 x 32 x 4096 78.1 -> 77.9.
template <int KCH, int STAGES, int G, int TILES, int DC>
__global__ void __launch_bounds__(kc::max_warps(G) * 32, 1) k_compute_kernel(const __grid_constant__ KParams p) {
    using namespace kc;
    constexpr int F_TILE = f_tile(KCH, TILES), N_TILE = n_tile(KCH, TILES);
    constexpr int F_BYTES = TILES * F_TILE, N_BYTES = TILES * N_TILE, STAGE = F_BYTES + 2 * N_BYTES;
    constexpr int F_IT = KCH / 8;                 // 16-byte copies per lane and tile for the high-byte plane
    constexpr int ROW_LANES = 2 * KCH;            // lanes that cover the nibble rows of one tile
    constexpr int TILES_PER_IT = 32 / ROW_LANES;  // 1 (KCH 16) or 2 (KCH 8)
    constexpr int N_IT = (TILES + TILES_PER_IT - 1) / TILES_PER_IT;
    static_assert((KCH == 8 || KCH == 16) && (TILES == 1 || TILES == 4), "channels per stage, tiles per unit");
    extern __shared__ __align__(128) uint8_t smem[];
    pdl_trigger();
    if (!p.k_exp) pdl_wait();
    const int D = DC ? DC : p.D;
    constexpr int NR = DC ? (DC + 31) / 32 : MAX_D / 32;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int wpc = blockDim.x >> 5;
    const int w = blockIdx.x * wpc + warp;
    const int u_begin = w * p.upw;
    if (u_begin >= p.units) {
        if (p.k_exp) pdl_wait();
        return;
    }
    const int u_end = (u_begin + p.upw < p.units) ? u_begin + p.upw : p.units;
    const int nch = D / KCH;
    const int total = (u_end - u_begin) * nch;
    const size_t tile_f = (size_t)D * 64, tile_n = (size_t)D * 32;
    const int META = meta_bytes(D, G), HMETA = head_meta(D, G);

    uint8_t* ring = smem + (size_t)warp * (STAGES * STAGE + META);
    uint8_t* meta0 = ring + STAGES * STAGE;
    uint8_t* tables = meta0 + 2 * MASK_BYTES;
    const uint32_t ring_a = smem_u32(ring);

    auto cursor_at = [&](int u) {
        KCursor k;
        k.u = u;
        k.bh = u / p.ngroups;
        k.g = u - k.bh * p.ngroups;
        k.c = 0;
        k.slot = 0;
        k.row = ((size_t)k.bh * p.nmb + (size_t)k.g * TILES) * D;
        return k;
    };
    auto advance = [&](KCursor& k) {   // next stage; returns true when a new (batch, KV head) starts
        k.row += KCH;
        if (++k.c < nch) return false;
        k.c = 0;
        ++k.u;
        if (++k.g < p.ngroups) {
            k.row += (size_t)(TILES - 1) * D;          // next tiles of the same (batch, KV head)
            return false;
        }
        k.g = 0;
        ++k.bh;
        k.slot ^= 1;
        k.row = (size_t)k.bh * p.nmb * D;
        return true;
    };
    auto load_masks = [&](long long bh, int slot) {
        uint32_t* um = reinterpret_cast<uint32_t*>(meta0 + slot * MASK_BYTES);
        uint32_t* table = reinterpret_cast<uint32_t*>(tables + slot * HMETA);
        kc_load_masks<G, NR>(p, bh, um, table, lane);
    };
    auto load_tables = [&](long long bh) {
        if (G > 1) kc_load_tables<G, NR>(p, bh, tables, lane);
    };

    const int nrow = (lane % ROW_LANES) >> 1, nhalf = (lane & 1) << 4, ntsub = lane / ROW_LANES;

    // ---- producer: async copies of one stage
    KCursor pk = cursor_at(u_begin);
    int pstage = 0;
    auto issue = [&]() {
        const uint32_t* masks = reinterpret_cast<const uint32_t*>(meta0 + pk.slot * MASK_BYTES);
        const int sh = ((pk.c * KCH) & 31) + nrow, wi = (pk.c * KCH) >> 5;
        const bool need_m = (masks[wi] >> sh) & 1u;
        const bool need_l = (masks[8 + wi] >> sh) & 1u;
        const uint32_t st = ring_a + (uint32_t)pstage * STAGE;
        const int ptiles = p.nb - pk.g * TILES;
        const uint8_t* pf = p.first8 + pk.row * 64 + lane * 16;
        const size_t pn = (pk.row + nrow) * 32 + nhalf;
        const uint8_t *pm = p.mid4 + pn, *pl = p.last4 + pn;
        const uint32_t fd = st + lane * 16, nd = st + F_BYTES + nrow * 32 + nhalf;
        auto copies = [&](auto whole) {                      // whole: all tiles of the unit exist
            constexpr bool WHOLE = decltype(whole)::value;
#pragma unroll
            for (int it = 0; it < TILES * F_IT; ++it) {      // high-byte plane: KCH*64 contiguous bytes per tile
                const int t = it / F_IT, v = it % F_IT;
                if (WHOLE || t < ptiles) cp_async16(fd + t * F_TILE + v * 512, pf + t * tile_f + v * 512);
            }
#pragma unroll
            for (int it = 0; it < N_IT; ++it) {              // nibble planes: only the rows some head reads
                const int t = it * TILES_PER_IT + ntsub;
                if ((WHOLE && TILES_PER_IT == 1) || (t < ptiles && t < TILES)) {
                    const uint32_t dm = nd + t * N_TILE, dl = dm + N_BYTES;
                    if (need_m) cp_async16(dm, pm + t * tile_n);
                    else if (G == 1) st_shared_v4(dm, 0x88888888u);              // plane not read: low byte becomes 0x80
                    if (need_l) cp_async16(dl, pl + t * tile_n);
                    else if (G == 1) st_shared_v4(dl, need_m ? 0x88888888u : 0u);  // low plane not read: low nibble becomes 8
                }
            }
        };
        if (ptiles >= TILES) copies(std::true_type{});
        else copies(std::false_type{});
        pstage = (pstage + 1 == STAGES) ? 0 : pstage + 1;
        if (advance(pk) && pk.u < u_end) load_masks(pk.bh, pk.slot);
    };

    // ---- prologue
    load_masks(pk.bh, 0);
    for (int j = 0; j < STAGES - 1; ++j) {
        if (j < total) issue();
        cp_async_commit();
    }
    const int tile = lane / (32 / TILES), li = lane % (32 / TILES);
    uint32_t acc[G][TILES];
#pragma unroll
    for (int g = 0; g < G; ++g)
#pragma unroll
        for (int j = 0; j < TILES; ++j) acc[g][j] = 0;
    KCursor ck = cursor_at(u_begin);
    load_tables(ck.bh);
    int cstage = 0;
    for (int i = 0; i < total; ++i) {
        cp_async_wait<STAGES - 2>();
        __syncwarp();
        if (i + STAGES - 1 < total) issue();
        cp_async_commit();

        const uint8_t* stp = ring + (size_t)cstage * STAGE;
        cstage = (cstage + 1 == STAGES) ? 0 : cstage + 1;
        const uint8_t* fp = stp + tile * F_TILE + li * 2 * TILES;
        const uint8_t* mp = stp + F_BYTES + tile * N_TILE + li * TILES;
        const uint8_t* lp = mp + N_BYTES;
        const uint8_t* hm0 = tables + (G == 1 ? ck.slot * HMETA : 0);
        const int ch0 = ck.c * KCH;                       // first channel of the stage
        if (G == 1) {
#pragma unroll
            for (int r4 = 0; r4 < KCH / 4; ++r4) {
                const uint4 qv = *reinterpret_cast<const uint4*>(hm0 + (size_t)(ch0 + r4 * 4) * 4);
#pragma unroll
                for (int rr = 0; rr < 4; ++rr) {
                    // the producer has written the substitutes into the rows it did not fetch
                    const int r = r4 * 4 + rr;
                    uint32_t wd[TILES];
                    kc_row<TILES>(wd, fp + r * 64, mp + r * 32, lp + r * 32);
                    const uint32_t q2 = u4w(qv, rr);
#pragma unroll
                    for (int j = 0; j < TILES; ++j) acc[0][j] = hfma2_bits(wd[j], q2, acc[0][j]);
                }
            }
        } else {
#pragma unroll
            for (int r4 = 0; r4 < KCH / 4; ++r4) {
                uint4 mk[G], cn[G];
                uint2 qv[G];
#pragma unroll
                for (int g = 0; g < G; ++g) {
                    const uint8_t* hg = hm0 + (size_t)g * HMETA + (size_t)(ch0 + r4 * 4) * 4;
                    mk[g] = *reinterpret_cast<const uint4*>(hg);
                    cn[g] = *reinterpret_cast<const uint4*>(hg + (size_t)D * 4);
                    qv[g] = *reinterpret_cast<const uint2*>(hm0 + (size_t)g * HMETA + (size_t)D * 8 + (size_t)(ch0 + r4 * 4) * 2);
                }
#pragma unroll
                for (int rr = 0; rr < 4; ++rr) {
                    const int r = r4 * 4 + rr;
                    uint32_t wd[TILES];
                    kc_row<TILES>(wd, fp + r * 64, mp + r * 32, lp + r * 32);
#pragma unroll
                    for (int g = 0; g < G; ++g) {
                        const uint32_t m = u4w(mk[g], rr), c = u4w(cn[g], rr), qw = rr < 2 ? qv[g].x : qv[g].y;
                        const __half2 q2 = kc_dup(qw, rr & 1);
#pragma unroll
                        for (int j = 0; j < TILES; ++j) acc[g][j] = kc_fma((wd[j] & m) | c, q2, acc[g][j]);
                    }
                }
            }
        }
        const long long cbh = ck.bh;
        const int cg = ck.g;
        const bool last_chunk = (ck.c == nch - 1);
        if (advance(ck) && ck.u < u_end) load_tables(ck.bh);
        if (last_chunk) {  // unit finished: scale, reorder to token order, one store per lane and head
            const int blk = cg * TILES + tile;
#pragma unroll
            for (int g = 0; g < G; ++g) {
                if (blk < p.nb) {
                    uint32_t a[TILES];
#pragma unroll
                    for (int j = 0; j < TILES; ++j) a[j] = hmul2_bits(acc[g][j], p.scale2);
                    const size_t row = (size_t)(cbh * G + g) * (size_t)(p.nb + 1) * 64 + (size_t)blk * 64 + li * 2 * TILES;
                    uint8_t* dst = p.s + row * 2;
                    if (TILES == 4)
                        *reinterpret_cast<uint4*>(dst) = make_uint4(__byte_perm(a[0], a[1 % TILES], 0x5410), __byte_perm(a[0], a[1 % TILES], 0x7632),
                                                                    __byte_perm(a[2 % TILES], a[3 % TILES], 0x5410),
                                                                    __byte_perm(a[2 % TILES], a[3 % TILES], 0x7632));
                    else *reinterpret_cast<uint32_t*>(dst) = a[0];
                }
#pragma unroll
                for (int j = 0; j < TILES; ++j) acc[g][j] = 0;
            }
        }
    }
    cp_async_wait<0>();
    if (p.k_exp) pdl_wait();
}

// Any block length / head size: one thread per token, planes read straight from global memory.
__global__ void __launch_bounds__(128)
k_compute_generic_kernel(const uint8_t* __restrict__ first8, const uint8_t* __restrict__ mid4,
                         const uint8_t* __restrict__ last4, const uint8_t* __restrict__ kq,
                         const uint8_t* __restrict__ kqmax, const __half* __restrict__ q, __half* __restrict__ s,
                         int nb, int nmb, int D, int d_block, int G, __half scale, int reference, long long total) {
    const int hb = d_block >> 1;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        int t = (int)(i % d_block);
        long long r = i / d_block;
        int z = (int)(r % nb);
        long long bh = r / nb;            // (batch, query head)
        const long long bkv = bh / G;     // (batch, KV head)
        const uint32_t top = kqmax[bh];
        __half acc = __ushort_as_half(0);
        for (int d = 0; d < D; ++d) {
            uint32_t diff = (top - (uint32_t)kq[bh * D + d]) & 0xFFu;
            long long row = ((bkv * nmb + z) * D + d) * hb;
            uint32_t f = first8[2 * row + t];
            uint32_t mb = 0x88u, lb = 0x00u;
            if (reference || diff < 8) {
                mb = mid4[row + (t >> 1)];
                lb = (reference || diff < 4) ? (uint32_t)last4[row + (t >> 1)] : 0x88u;
            }
            uint32_t bits = (t & 1) ? ((f << 8) + ((mb & 0x0Fu) << 4) + (lb & 0x0Fu))
                                    : ((f << 8) + (mb & 0xF0u) + ((lb & 0xF0u) >> 4));
            acc = __hfma(__ushort_as_half((unsigned short)bits), q[bh * D + d], acc);
        }
        s[bh * (long long)(nb + 1) * d_block + (long long)z * d_block + t] = __hmul(acc, scale);
    }
}

// Whether launch_k_compute takes the streaming kernel, which can make the alignment inputs itself.
static bool k_fast(const uint8_t* first8, const uint8_t* mid4, const uint8_t* last4, const uint8_t* kq, const uint8_t* q,
                   const uint8_t* s, int group, int D, int d_block) {
    return d_block == 64 && D % 16 == 0 && D >= 64 && D <= kc::MAX_D && aligned16(first8) && aligned16(mid4) &&
           aligned16(last4) && aligned16(kq) && aligned16(q) && aligned16(s) &&
           (group == 1 || group == 2 || group == 4 || group == 8);
}
bool k_compute_aligns(const uint8_t* first8, const uint8_t* mid4, const uint8_t* last4, const uint8_t* kq, const uint8_t* q,
                      const uint8_t* s, int group, int D) {
    return k_fast(first8, mid4, last4, kq, q, s, group, D, 64);
}

// Launch of one form: warps per CTA and units per warp, one CTA per SM.
template <int KCH, int STAGES, int G, int TILES, int DC = 0>
static int k_launch(KParams p, cudaStream_t st) {
    using namespace kc;
    p.ngroups = (p.nb + TILES - 1) / TILES;
    const long long units = (long long)p.BH * p.ngroups;
    AKV_REQUIRE(units < (1ll << 30), AKV_ERR_OVERFLOW, "k_cache_compute: too many blocks");
    p.units = (int)units;
    const int sms = sm_count(), budget = max_dyn_smem();
    const int per_warp = STAGES * stage_bytes(KCH, TILES) + meta_bytes(p.D, G);
    int wmax = budget / per_warp;
    if (wmax > max_warps(G)) wmax = max_warps(G);
    if (tuning().k_wpc > 0 && tuning().k_wpc < wmax) wmax = tuning().k_wpc;
    AKV_REQUIRE(wmax >= 1, AKV_ERR_CUDA, "k_cache_compute: %d bytes of shared memory are too few", budget);
    // (fewer units than that: spread over the SMs first, a warp streams the faster the fewer share its SM)
    if (units < (long long)sms * wmax) wmax = (int)((units + sms - 1) / sms);
    // Trim the warp count so that every warp gets (nearly) the same whole number of units.
    int wpc = wmax;
    double best_eff = -1.0;
    for (int c = wmax; c >= (wmax * 3 + 3) / 4; --c) {
        long long Wt = (long long)sms * c;
        long long upw = (units + Wt - 1) / Wt;
        double eff = (double)units / (double)(upw * Wt);
        if (eff > best_eff + 0.02) { best_eff = eff; wpc = c; }
    }
    {
        long long Wt = (long long)sms * wpc;
        p.upw = (int)((units + Wt - 1) / Wt);
    }
    const long long warps_needed = (units + p.upw - 1) / p.upw;
    const int grid = (int)((warps_needed + wpc - 1) / wpc);
    // the opt-in shared-memory size is a per-device attribute of the kernel: set once per device - to the device's maximum, so
    // that every launch shape fits - not on every launch (a racing thread at worst sets it twice)
    static std::atomic<bool> configured[64];
    const auto kern = k_compute_kernel<KCH, STAGES, G, TILES, DC>;
    int dev = -1;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !configured[dev].load(std::memory_order_acquire)) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, budget);
        if (e != cudaSuccess) return cuda_status(e, "k_cache_compute smem attribute");
        if (dev >= 0 && dev < 64) configured[dev].store(true, std::memory_order_release);
    }
    launch_chained(kern, dim3(grid), dim3(wpc * 32), (size_t)wpc * per_warp, st, p);
    return cuda_status(cudaGetLastError(), "k_cache_compute launch");
}

// q.K^T over nb quantized blocks.  H = KV heads, group = query heads per KV head; kq, kqmax, q and the score rows are
// per (batch, query head) with query head = KV head * group + g.  k_exp != nullptr (only when k_compute_aligns() holds and the
// kernel launched before is a pdl_turn one that writes no planes): the kernel makes kq and kqmax for itself from q, k_exp and the
// token k_new (or null), and runs beside that kernel.
int launch_k_compute_align(const uint8_t* first8, const uint8_t* mid4, const uint8_t* last4, const uint8_t* kq,
                           const uint8_t* kqmax, const uint8_t* q, uint8_t* s, int bsz, int H, int group, int nb, int nmb,
                           int D, int d_block, float sqrt_dim, int reference, const uint8_t* k_exp, const uint16_t* k_new,
                           cudaStream_t st) {
    using namespace kc;
    const __half scale = __float2half_rn(sqrt_dim);
    if (!k_fast(first8, mid4, last4, kq, q, s, group, D, d_block)) {
        AKV_REQUIRE(!k_exp, AKV_ERR_SHAPE, "k_cache_compute: the aligning form needs the streaming kernel");
        long long total = (long long)bsz * H * group * nb * d_block;
        long long want = (total + 127) / 128;
        int grid = (int)(want < (long long)sm_count() * 16 ? want : (long long)sm_count() * 16);
        count_launch();
        k_compute_generic_kernel<<<grid, 128, 0, st>>>(first8, mid4, last4, kq, kqmax,
                                                       reinterpret_cast<const __half*>(q),
                                                       reinterpret_cast<__half*>(s), nb, nmb, D, d_block, group,
                                                       scale, reference, total);
        return cuda_status(cudaGetLastError(), "k_cache_compute launch");
    }
    KParams p;
    p.first8 = first8; p.mid4 = mid4; p.last4 = last4; p.kq = kq; p.kqmax = kqmax; p.q = q; p.s = s;
    p.BH = bsz * H; p.nb = nb; p.nmb = nmb; p.D = D;
    p.ngroups = p.units = p.upw = 0;
    const unsigned short sb = __half_as_ushort(scale);
    p.scale2 = (uint32_t)sb | ((uint32_t)sb << 16);
    p.reference = reference;
    p.k_exp = k_exp;
    p.k_new = k_new;

    // Units of one tile for groups of four and eight heads while there are at most four tiles per SM: many short chains of
    // stages instead of few long ones, their whole depth of channels in flight.  A decode step in us, four tiles against one:
    // 8 KV heads x 4, batch 1, 700 tokens (80 tiles) 31.8 / 27.0, 4096 tokens (512) 47.6 / 42.8; 4 x 8, 8000 tokens (500)
    // 78.1 / 69.9; 2000 tiles 67.2 / 75.6.  One head: 384 tiles 25.1 / 24.9, 800 26.7 / 25.9, 1472 26.8 / 29.2.
    const bool single = tuning().k_tiles ? tuning().k_tiles == 1 : (long long)p.BH * nb <= 4ll * sm_count();
    const bool d128 = D == 128;
    if (single && D >= 128 && group == 4) return d128 ? k_launch<16, 8, 4, 1, 128>(p, st) : k_launch<16, 8, 4, 1>(p, st);
    if (single && D >= 128 && group == 8) return d128 ? k_launch<16, 8, 8, 1, 128>(p, st) : k_launch<16, 8, 8, 1>(p, st);
    // (channels per stage, ring depth): the instantiated combinations; anything else falls back to the default of its group
    if (group == 1) {
        const int kch = tuning().k_kch;
        int stages = tuning().k_stages;
        if (!((kch == 8 && (stages == 3 || stages == 4 || stages == 6)) || (kch == 16 && stages >= 3 && stages <= 5)))
            stages = (kch == 8) ? 4 : 3;
        if (stages > D / kch) stages = D / kch;      // (D >= 64: four stages of 16 channels)
        switch (kch * 10 + stages) {
            case 83: return k_launch<8, 3, 1, 4>(p, st);
            case 84: return k_launch<8, 4, 1, 4>(p, st);
            case 86: return k_launch<8, 6, 1, 4>(p, st);
            case 164: return k_launch<16, 4, 1, 4>(p, st);
            case 165: return k_launch<16, 5, 1, 4>(p, st);
            case 163: return d128 ? k_launch<16, 3, 1, 4, 128>(p, st) : k_launch<16, 3, 1, 4>(p, st);
            default:
                set_error("k_cache_compute: no kernel for %d channels x %d stages", kch, stages);
                return AKV_ERR_SHAPE;
        }
    }
    if (group == 2) return d128 ? k_launch<gqa_kch(2), gqa_stages(2), 2, 4, 128>(p, st)
                                : k_launch<gqa_kch(2), gqa_stages(2), 2, 4>(p, st);
    if (group == 4) return d128 ? k_launch<gqa_kch(4), gqa_stages(4), 4, 4, 128>(p, st)
                                : k_launch<gqa_kch(4), gqa_stages(4), 4, 4>(p, st);
    return d128 ? k_launch<gqa_kch(8), gqa_stages(8), 8, 4, 128>(p, st)
                : k_launch<gqa_kch(8), gqa_stages(8), 8, 4>(p, st);
}

int launch_k_compute(const uint8_t* first8, const uint8_t* mid4, const uint8_t* last4, const uint8_t* kq,
                     const uint8_t* kqmax, const uint8_t* q, uint8_t* s, int bsz, int H, int group, int nb, int nmb,
                     int D, int d_block, float sqrt_dim, int reference, cudaStream_t st) {
    return launch_k_compute_align(first8, mid4, last4, kq, kqmax, q, s, bsz, H, group, nb, nmb, D, d_block, sqrt_dim,
                                  reference, nullptr, nullptr, st);
}

}  // namespace akv

// Exact-order P.V: the kernel body behind v_cache_compute for head_dim 128.
//
// Replaces the reference's v_cache_compute_kernel (extension/csrc/V_cache.cu:178-308); bit-identical outputs: every
// output channel is the fp16 fused-multiply-add chain over tokens 0..n-1 in order (V_cache.cu:203,304), skipped nibble
// planes are replaced by the reference's constants (V_cache.cu:198-202,250-253).
//
// Design (B200).  The token order leaves one dependent chain per (batch, query head, channel pair), and the V layout is
// token-major (a token's 128 high bytes are one row) while a chain thread wants "my channel pairs, next tokens".  That
// transposition is done by the load instruction: ldmatrix.x4.trans over eight token rows (one 8x8 matrix of 16-bit words
// per two tokens: four 16-byte chunks of each, the warp's half of the channels) hands lane T, for each two tokens, one
// register holding their high-byte pairs of channel pair 32*half + 8*(T%4) + T/4.  The two tokens' chunks lie 128 bytes
// apart, in the same banks: a two-way conflict on every one of these loads.
// A token that reads no nibble plane - the rule - has the constant low byte 0x80, so its two fp16 words are two byte
// permutes of that register, the same for every query head of the KV head: a chain warp runs the chains of GH heads, per
// token two permutes and 2 GH FMAs.
//   A unit = the query heads of one (batch, KV head), or one of them (while they are few the heads of a KV head do better
//   with rings of their own: they stream the same planes at the same pace and meet in L2): a ring of 64-token stages in shared memory, W = NH / GH chain warps that drain it and HW
//   helper warps that fill it (stage i belongs to helper i % HW).  A CTA holds UPC units (warps ordered so that the chain
//   warps lie on different schedulers); with more units than fit at once a (helpers, chains) group walks through several
//   of them without draining its ring.
//   A stage = 8 KB of high bytes as they lie in the plane (one bulk copy), the probabilities of the unit's heads, and per
//   head and token the place of the token's 128 LOW bytes: a constant row of 0x80, or, for a token that reads a nibble
//   plane, a row of the helper's pool, built for the token's code.  Low bytes are fetched like the high ones - every
//   lane of an ldmatrix names the row it loads, so a token's row can lie anywhere - which keeps the chain's instruction
//   stream straight whatever the codes are.  Stages without a flagged token run a second copy of the body that does not
//   fetch low bytes; that is the only branch.  It matters: a taken branch costs a lone warp tens of cycles, and forms
//   that branched to other code for groups of 8 tokens with a flagged one lost more on the 1 % of flagged tokens than the
//   rest gained.
//   helper warp: lane = tokens (2 lane, 2 lane + 1) of its stage.  Waits for the slot to be released, starts the high
//     bytes' copy, takes the heads' probabilities (loaded from global memory a stage of its own ahead) and decides the
//     read codes (V_cache.cu:211,250-251); then it finishes its PREVIOUS stage (builds the rows from the nibble rows
//     requested an iteration ago, arrives), hands out pool rows for this stage, stores probabilities and places and
//     requests the nibble rows.  An iteration is a chain of latencies of 700 to 1500 cycles, several times what the chains
//     need for a stage: hence several helpers.
// What bounds it: with two units on every SM the high bytes' stream from HBM and the FMA pipe (an fp16x2 FMA issues every
// other cycle: 4 heads are 16 cycles per token), with few units the chain: 6 to 7 cycles per token.
// Every wait is bounded (about a second); a wait that runs out raises the device error flag, the chain stores NaN
// instead of a result, and the helper gives its copies in flight time to land before the CTA leaves.
#pragma once
#include "akv_common.cuh"

namespace akv {

struct VParams {
    const uint8_t* first8;
    const uint8_t* mid4;
    const uint8_t* last4;
    const uint16_t* s;      // probabilities, one row per (batch, query head)
    const uint8_t* amin;    // threshold byte per (batch, query head)
    // test_o != nullptr: the kernel computes the threshold bytes itself from the probe result [B,Hq,D] and the
    // exponent maxima [B,H,D] (v_threshold_warp) and stores them to amin_out
    const uint16_t* test_o;
    const uint8_t* v_exp;
    uint8_t* amin_out;
    int H;                  // KV heads
    uint16_t* o;            // [B, Hq, D]
    int max_seq_len, D, s_last_dim, n, reference;
    int group;              // query heads per KV head (1 = multi-head attention)
    int nf;                 // chain kernel: ring depth (stages)
    int units;              // chain kernel: number of units
    int share;              // chain kernel: units that read the planes of one KV head (group / heads per unit)
    // chain kernel: res != nullptr adds the residual tokens' part of the output, [B, Hq, D] fp16 computed by the
    // softmax kernel: out = half(o + res) (extension/v_cache_file.py:189), which saves the tail launch
    const uint16_t* res;
    // chain kernel: the kernel launched before is a pdl_turn one that writes no planes: their first stages are requested before
    // it has completed
    int early;
};

// ---- device error flag and shared-memory barriers (mbarrier) with bounded waits
static __device__ unsigned int g_v_wait_gave_up = 0;   // set when a bounded wait ran out (never expected)

__device__ __forceinline__ void mbar_init(uint32_t a, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(a), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t a) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(a) : "memory");
}
// arrives and adds `bytes` to the byte count the current phase still waits for
__device__ __forceinline__ void mbar_arrive_expect(uint32_t a, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(a), "r"(bytes) : "memory");
}
// Bounded wait, split so that the common case (the phase has completed, or completes within the hardware's own short
// wait) is a single instruction in the caller's instruction stream and the spin loop lives out of line: the loops that
// call this are latency-critical and must stay compact in the instruction cache.
__device__ __noinline__ bool mbar_wait_slow(uint32_t a, uint32_t parity) {
    unsigned long long t0 = 0;
    for (int spin = 0; spin < (1 << 26); ++spin) {
        uint32_t ok;
        // the hint lets the hardware park the warp (no issue slots taken from the warps that share its scheduler)
        // until the phase completes or the time (ns) runs out
        asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\nselp.u32 %0, 1, 0, p;\n}\n"
                     : "=r"(ok) : "r"(a), "r"(parity), "r"(20000u) : "memory");
        if (ok) return true;
        if ((spin & 63) == 63) {
            unsigned long long t;
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
            if (t0 == 0) t0 = t;
            else if (t - t0 > 1000000000ull) break;      // about a second: give up and raise the device error flag
        }
    }
    atomicOr(&g_v_wait_gave_up, 1u);
    return false;
}
__device__ __forceinline__ bool mbar_wait(uint32_t a, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(ok) : "r"(a), "r"(parity) : "memory");
    if (__builtin_expect(ok != 0, 1)) return true;
    return mbar_wait_slow(a, parity);
}
// Bulk asynchronous copy global -> shared through the TMA unit; 16-byte aligned addresses, size a multiple of 16.
// Completion is signalled on the mbarrier as `bytes` of its pending byte count.
__device__ __forceinline__ void bulk_copy(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}

namespace vch {
constexpr int D = 128, HD = 64;    // head size, bytes of a nibble row
constexpr int TOK = 64;            // tokens per stage
// Helper warps per unit (the ring depth is a multiple: a slot's stages all belong to one helper).  Four, or two where the
// pools of four would leave too little room for the ring.  (Stages of 128 tokens, prepared by two helpers, were faster in
// back-to-back launches and slower in a decode step, where every plane byte comes from HBM: 96 against 85 us per step at
// batch 8 x 32 heads x 4096 tokens.)
// Two units of two heads: three, with a ring of six stages (two with eight were what the chains waited for: 24 sequences x 16 KV
// heads x 2 x 8192 tokens 302 -> 271 us per step, 32 x 16 x 2 x 4096 204 -> 184; units of four heads do not gain, 480 / 480).
__host__ __device__ constexpr int helpers(int upc, int heads) {
    return upc > (heads > 1 ? 1 : 2) ? (heads == 2 ? 3 : 2) : 4;
}
// A ring slot: high bytes | probabilities [heads][TOK] | places of the low bytes [heads][8][8] (token 8 g + w of the
// stage at [w][g]: what a lane needs for its rows of the groups lies together), in 2-byte units into the unit's pools |
// how many tokens of the stage read a nibble plane
__host__ __device__ constexpr int off_s() { return TOK * D; }
__host__ __device__ constexpr int off_low(int heads) { return off_s() + heads * TOK * 2; }
__host__ __device__ constexpr int off_any(int heads) { return off_low(heads) + heads * TOK * 2; }
__host__ __device__ constexpr int slot_bytes(int heads) { return (off_any(heads) + 4 + 127) & ~127; }
// Rows of a helper's pool: a token has one code with one head per unit, up to two (both planes; mid only) with several;
// all tokens of a stage must fit at once.
__host__ __device__ constexpr int rows_per_token(int heads) { return heads > 1 ? 2 : 1; }
__host__ __device__ constexpr int pool_rows(int heads) { return TOK * rows_per_token(heads); }
// A unit's share of the shared memory: nf slots | the helpers' pools and the constant row | per helper the list of a
// stage's flagged tokens | pool position after each slot's stage | barriers full[nf], free[nf]
struct Plan {
    int pool, list, cum, bar, bytes;
};
__host__ __device__ constexpr Plan plan(int nf, int upc, int heads) {
    Plan p{};
    const int hw = helpers(upc, heads);
    p.pool = nf * slot_bytes(heads);
    p.list = p.pool + (hw * pool_rows(heads) + 1) * D;
    p.cum = p.list + hw * TOK * 2;
    p.bar = (p.cum + nf * 4 + 7) & ~7;
    p.bytes = (p.bar + 2 * nf * 8 + 127) & ~127;
    return p;
}
}  // namespace vch

// Both halves of the result = half `hi ? 1 : 0` of w (the probability of one token for both channels of a pair).
__device__ __forceinline__ __half2 v_dup(uint32_t w, int hi) {
    const __half2 h = *reinterpret_cast<const __half2*>(&w);
    return hi ? __high2half2(h) : __low2half2(h);
}
__device__ __forceinline__ uint32_t v_fma(uint32_t k, __half2 s, uint32_t acc) {
    const __half2 r = __hfma2(*reinterpret_cast<const __half2*>(&k), s, *reinterpret_cast<const __half2*>(&acc));
    return *reinterpret_cast<const uint32_t*>(&r);
}

// About a millisecond of sleep: after a wait gave up (never expected), the copies in flight get time to land before
// the CTA's shared memory is released.
__device__ __noinline__ void v_sleep_ms() {
#pragma unroll 1
    for (int k = 0; k < 1000; ++k) __nanosleep(1000);
}

__device__ __forceinline__ uint4 v_ldg128(const void* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ void sts128(uint32_t a, const uint4& v) {
    asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};\n" ::"r"(a), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ void sts32(uint32_t a, uint32_t v) { asm volatile("st.shared.u32 [%0], %1;\n" ::"r"(a), "r"(v) : "memory"); }
__device__ __forceinline__ void sts16(uint32_t a, uint32_t v) {
    asm volatile("st.shared.u16 [%0], %1;\n" ::"r"(a), "h"((uint16_t)v) : "memory");
}

// 32 low bytes of a token (16 channel pairs) from 16 bytes of its mid and low plane rows.  A pair's byte holds the even
// channel's nibble above the odd one's; the even channel's low byte is mid.hi:low.hi, the odd one's mid.lo:low.lo
// (V_cache.cu:250-253).
__device__ __forceinline__ void v_low_bytes(uint32_t dst, const uint4& m, const uint4& l) {
    uint32_t o[8];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const uint32_t mw = u4w(m, j), lw = u4w(l, j);
        const uint32_t ev = (mw & 0xF0F0F0F0u) | ((lw >> 4) & 0x0F0F0F0Fu), od = ((mw << 4) & 0xF0F0F0F0u) | (lw & 0x0F0F0F0Fu);
        o[2 * j] = __byte_perm(ev, od, 0x5140);
        o[2 * j + 1] = __byte_perm(ev, od, 0x7362);
    }
    sts128(dst, make_uint4(o[0], o[1], o[2], o[3]));
    sts128(dst + 16, make_uint4(o[4], o[5], o[6], o[7]));
}

// NH query heads per unit, GH of them per chain warp, UPC units per CTA at a time.
template <int NH, int GH, int UPC>
__global__ void __launch_bounds__(UPC * (2 * NH / GH + vch::helpers(UPC, NH)) * 32, 1) v_chain_kernel(const VParams p) {
    using namespace vch;
    extern __shared__ __align__(128) uint8_t smem[];
    constexpr int W = 2 * NH / GH, HW = helpers(UPC, NH), NG = TOK / 8;
    constexpr int SLOT = slot_bytes(NH), RPT = rows_per_token(NH), NP = pool_rows(NH);
    constexpr int OFF_S = off_s(), OFF_LOW = off_low(NH), OFF_ANY = off_any(NH);
    constexpr uint32_t CONST_ROW = HW * NP * D;    // place of the constant low bytes
    const int lane = threadIdx.x & 31, wcta = threadIdx.x >> 5;
    // warps: the chain warps of all units first (consecutive warps go to different schedulers), then the helpers
    const bool helper = wcta >= UPC * W;
    const int uc = helper ? (wcta - UPC * W) / HW : wcta / W;
    const int wi = helper ? wcta - UPC * W - uc * HW : wcta - uc * W;      // warp inside the unit's helpers / chains
    const int nf = p.nf, n = p.n, nst = (n + TOK - 1) / TOK;
    const Plan pl = plan(nf, UPC, NH);
    const uint32_t ring = smem_u32(smem) + (uint32_t)(uc * pl.bytes);
    const uint32_t pool = ring + pl.pool, bar_full = ring + pl.bar, bar_free = bar_full + nf * 8;
    if (helper) {
        if (wi == 0 && lane == 0) {
            for (int s = 0; s < nf; ++s) {
                mbar_init(bar_full + s * 8, 2);    // the high bytes' copy and the helper's arrival
                mbar_init(bar_free + s * 8, W);    // the chain warps
            }
            asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        }
        sts32(pool + CONST_ROW + lane * 4, 0x80808080u);
    }
    pdl_trigger();
    if (!p.early) pdl_wait();
    __syncthreads();
    // units are dealt out a grid apart, so that every SM gets its share
    const int first_unit = uc * gridDim.x + blockIdx.x, stride = UPC * gridDim.x;
    const int nunits = first_unit < p.units ? (p.units - first_unit + stride - 1) / stride : 0;   // of this group

    if (helper) {
        // ------------------------------------------------------------------ helper warp
        // Its stages are q = wi, wi + HW, ... of the group's stages 0 .. nunits * nst - 1; stage q uses slot q % nf.
        const uint32_t list = ring + pl.list + wi * TOK * 2, cum = ring + pl.cum;
        const uint32_t mine = (uint32_t)wi * NP * D;                       // place of the pool
        const long long total = (long long)nunits * nst;
        bool alive = true;
        int slot = wi;                             // of stage q (nf is a multiple of HW)
        int rel = wi, out = 0;                     // slot of its oldest stage whose release has not been consumed; stages since
        uint32_t rel_par = 0;                      // parity of that release
        uint32_t head = 0, tail = 0;               // pool rows handed out / taken back so far
        // consume the release of its oldest stage: the slot and the stage's pool rows are free again
        auto reclaim = [&]() {
            alive = mbar_wait(bar_free + rel * 8, rel_par);
            tail = lds32(cum + rel * 4);
            --out;
            if ((rel += HW) >= nf) { rel -= nf; rel_par ^= 1u; }
        };
        const int lim_m = p.reference ? 0x8000 : 0x0800, lim_l = p.reference ? 0x8000 : 0x0400;    // (0x8000: always)
        auto plane_row = [&](int unit) { return (size_t)(NH > 1 ? unit : unit / p.share) * p.max_seq_len; };   // of its token 0
        auto copy_high = [&](size_t row, int i, int sl) {
            const uint32_t bytes = (uint32_t)min(TOK, n - i * TOK) * D;
            mbar_arrive_expect(bar_full + sl * 8, bytes);
            bulk_copy(ring + (uint32_t)sl * SLOT, p.first8 + (row + (size_t)i * TOK) * D, bytes,
                      bar_full + sl * 8);
        };
        // the first ring's high bytes depend on nothing but the planes: under way before the thresholds are known
        const int early = min(nf, nst);
        if (nunits > 0 && wi + HW * lane < early) copy_high(plane_row(first_unit), wi + HW * lane, wi + HW * lane);
        if (p.early) pdl_wait();
        // the unit's thresholds; probabilities of this lane's two tokens of its next stage
        uint32_t A[NH], nxt[NH];
        auto load_s = [&](int unit, int i) {       // (rows are padded to a multiple of 8 values)
            const int t = i * TOK + 2 * lane;
#pragma unroll
            for (int g = 0; g < NH; ++g)
                nxt[g] = t < n ? *reinterpret_cast<const uint32_t*>(p.s + ((size_t)unit * NH + g) * p.s_last_dim + t) : 0u;
        };
        // the previous stage: its slot (-1: none), flagged tokens and their first pool row
        int pslot = -1, pcnt = 0;
        size_t ptok = 0;                           // plane row of its first token
        uint32_t prow = 0;
        // Nibble rows of eight flagged tokens, lane = (token lane/4, 16 bytes lane%4).  The stage's first AHEAD batches are
        // requested when it is prepared and turned into pool rows an iteration later, more of them NBT at a time.
        struct Batch {
            uint4 m, l;
            uint32_t t;                            // list entry: token | some head reads both planes << 8 | mid only << 9
        };
        auto request = [&](Batch& b, int k) {
            b.t = 0xFFFFu;
            if (8 * k + (lane >> 2) < pcnt) {
                b.t = lds16(list + (8 * k + (lane >> 2)) * 2);
                const size_t at = (ptok + (b.t & 0xFFu)) * HD + (lane & 3) * 16;
                b.m = v_ldg128(p.mid4 + at);
                if (b.t & 0x100u) b.l = v_ldg128(p.last4 + at);
            }
        };
        auto build = [&](const Batch& b, int k) {
            if (b.t == 0xFFFFu) return;
            const uint32_t r = (prow + (uint32_t)(8 * k + (lane >> 2)) * RPT) % NP;
            const uint32_t dst = pool + mine + r * D + (lane & 3) * 32;
            const uint4 c88 = make_uint4(0x88888888u, 0x88888888u, 0x88888888u, 0x88888888u);
            if (RPT == 1) {
                v_low_bytes(dst, b.m, b.t & 0x100u ? b.l : c88);
            } else {
                if (b.t & 0x100u) v_low_bytes(dst, b.m, b.l);
                if (b.t & 0x200u) v_low_bytes(dst + D, b.m, c88);    // (NP is even: the second row follows the first)
            }
        };
        constexpr int NBT = NH > 4 ? 4 : 8;        // (registers)
        // Batches requested when the stage is prepared (registers).  With one, a stage of flagged tokens waited for the loads of the
        // other seven (flat attention, batch 8 x 32 heads x 4096 tokens: 120 us per step, now 109).
        constexpr int AHEAD = NH > 1 ? 1 : UPC > 2 ? 4 : 8;
        Batch ahead[AHEAD];
#pragma unroll
        for (int j = 0; j < AHEAD; ++j) {
            ahead[j].m = ahead[j].l = make_uint4(0, 0, 0, 0);
            ahead[j].t = 0xFFFFu;
        }
        const int slots = nf / HW;                 // its share of the ring
        int unit = first_unit, i = wi;             // of stage q
        while (i >= nst && nst > 0 && unit < p.units) { i -= nst; unit += stride; }
        int aunit = -1;                            // the unit whose thresholds are in A
        size_t row = 0;                            // ... and the plane row of its token 0
        if (wi < total) load_s(unit, i);
#pragma unroll 1
        for (long long q = wi; q < total + HW && alive; q += HW) {
            const bool now = q < total;            // (else: only the previous stage is left)
            uint32_t cur[NH], code[NH], u0[2] = {0, 0}, u1[2] = {0, 0};   // even / odd tokens that read both planes / mid only for some head
            int nunit = unit, ni = i + HW;
            if (now) {
                const bool entered = aunit != unit;
                if (entered) {
                    aunit = unit;
                    row = plane_row(unit);
                }
                if (q >= early) {
                    while (alive && out >= slots) reclaim();
                    if (!alive) break;
                    if (lane == 0) copy_high(row, i, slot);
                }
                ++out;
                if (entered) {
#pragma unroll
                    for (int g = 0; g < NH; ++g) {
                        const long long bh = (long long)unit * NH + g;
                        uint32_t a;
                        if (p.test_o) {
                            a = v_threshold_warp(p.test_o, p.v_exp, bh, p.H, p.group, D, lane);
                            if (i == 0 && lane == 0) p.amin_out[bh] = (uint8_t)a;
                        } else {
                            a = p.amin[bh];
                        }
                        A[g] = (a << 10) & 0xFFFFu;
                    }
                }
#pragma unroll
                for (int g = 0; g < NH; ++g) cur[g] = nxt[g];
                while (ni >= nst) { ni -= nst; nunit += stride; }
                if (q + HW < total) load_s(nunit, ni);
                // read codes of this lane's tokens for every head: 16-bit wrap-around, signed compare
                // (V_cache.cu:211,250-251); a code is 0 when the token reads both planes, 1 mid only, 2 neither
                const int left = n - i * TOK - 2 * lane;     // of this lane's two tokens
                uint32_t r0 = 0, r1 = 0;                     // bit h: some head reads both planes / mid only
#pragma unroll
                for (int g = 0; g < NH; ++g) {
                    const int d0 = (int)(int16_t)(uint16_t)(A[g] - cur[g]), d1 = (int)(int16_t)(uint16_t)(A[g] - (cur[g] >> 16));
                    const uint32_t c0 = left < 1 || d0 >= lim_m ? 2u : d0 >= lim_l ? 1u : 0u;
                    const uint32_t c1 = left < 2 || d1 >= lim_m ? 2u : d1 >= lim_l ? 1u : 0u;
                    code[g] = c0 | c1 << 16;
                    r0 |= (c0 == 0 ? 1u : 0u) | (c1 == 0 ? 2u : 0u);
                    r1 |= (c0 == 1 ? 1u : 0u) | (c1 == 1 ? 2u : 0u);
                }
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    u0[h] = __ballot_sync(0xFFFFFFFFu, (r0 >> h) & 1u);
                    u1[h] = __ballot_sync(0xFFFFFFFFu, (r1 >> h) & 1u);
                }
            }
            // finish the previous stage
            if (pslot >= 0) {
                if (pcnt > 0) {
                    build(ahead[0], 0);
                    if (AHEAD > 1 && __builtin_expect(pcnt > 8, 0)) {
#pragma unroll
                        for (int j = 1; j < AHEAD; ++j) build(ahead[j], j);
                    }
#pragma unroll 1
                    for (int k = AHEAD; 8 * k < pcnt; k += NBT) {
                        Batch b[NBT];
#pragma unroll
                        for (int j = 0; j < NBT; ++j) request(b[j], k + j);
#pragma unroll
                        for (int j = 0; j < NBT; ++j) build(b[j], k + j);
                    }
                }
                __syncwarp();                      // (everything the lanes stored for this stage comes before the arrival)
                if (lane == 0) mbar_arrive(bar_full + pslot * 8);
            }
            if (!now) break;
            pslot = slot;
            ptok = row + (size_t)i * TOK;
            // pool rows and places of this stage
            const uint32_t sl = ring + (uint32_t)slot * SLOT;
            uint32_t place[2] = {CONST_ROW, CONST_ROW};
            pcnt = __popc(u0[0] | u1[0]) + __popc(u0[1] | u1[1]);
            if (pcnt != 0) {                       // (warp-uniform)
                // (its older stages have been armed, and the chains let go of them once the stage behind them - another
                // helper's - is there)
                while (alive && head + pcnt * RPT - tail > (uint32_t)NP) reclaim();
                if (!alive) break;
                prow = head % NP;
                head += pcnt * RPT;
                const uint32_t lt = (1u << lane) - 1u;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const uint32_t f = u0[h] | u1[h];
                    const int rank = (h ? __popc(u0[0] | u1[0]) : 0) + __popc(f & lt);
                    place[h] = mine + (prow + (uint32_t)rank * RPT) % NP * D;
                    if ((f >> lane) & 1u)
                        sts16(list + rank * 2, (2 * lane + h) | ((u0[h] >> lane) & 1u) << 8 | ((u1[h] >> lane) & 1u) << 9);
                }
                __syncwarp();
                request(ahead[0], 0);
                if (AHEAD > 1 && __builtin_expect(pcnt > 8, 0)) {
#pragma unroll
                    for (int j = 1; j < AHEAD; ++j) request(ahead[j], j);
                }
            }
#pragma unroll
            for (int g = 0; g < NH; ++g) sts32(sl + OFF_S + g * (TOK * 2) + lane * 4, cur[g]);
            if (pcnt != 0) {                       // (the places of other stages are not looked at)
#pragma unroll
                for (int g = 0; g < NH; ++g)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const uint32_t c = h ? code[g] >> 16 : code[g] & 0xFFFFu, t = 2 * lane + h;
                        const uint32_t at = c == 2 ? CONST_ROW : place[h] + (RPT == 2 && c == 1 ? D : 0);
                        sts16(sl + OFF_LOW + (g * TOK + (t & 7) * NG + (t >> 3)) * 2, at >> 1);
                    }
            }
            if (lane == 0) {
                sts32(sl + OFF_ANY, (uint32_t)pcnt);
                sts32(cum + slot * 4, head);
            }
            if ((slot += HW) >= nf) slot -= nf;
            unit = nunit;
            i = ni;
        }
        if (!alive) v_sleep_ms();
        return;
    }

    // ---------------------------------------------------------------------- chain warp
    constexpr int NB = GH <= 2 ? 4 : 2;            // groups of 8 tokens in flight
    const int half = wi & 1, h0 = (wi >> 1) * GH;                          // its channels and its first head
    const int pair = 32 * half + 8 * (lane & 3) + (lane >> 2);             // this lane's channel pair
    // row this lane names in an ldmatrix over a group of 8 tokens: matrix lane/8 = tokens 2 (lane/8) and the next, row
    // lane%8 = chunk (lane%8)/2 of the half, token (lane%8)%2
    const uint32_t lm_tok = 2 * (lane >> 3) + (lane & 1), lm_chunk = (4 * half + ((lane >> 1) & 3)) * 16;
    const uint32_t lm_off = lm_tok * D + lm_chunk, lm_low = pool + lm_chunk;
    const uint32_t s_off = OFF_S + h0 * TOK * 2, low_off = OFF_LOW + h0 * TOK * 2 + lm_tok * (NG * 2);
    // Registers of one group of 8 tokens: high bytes [even token's pair | odd token's pair], the heads' low bytes likewise,
    // and the heads' probabilities
    struct Grp {
        uint32_t h[4], l[GH][4];
        uint4 s[GH];
    };
    auto ldm = [](uint32_t* r, uint32_t a) {
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
    };
    auto fetch = [&](Grp& r, uint32_t sl, int grp) {
        ldm(r.h, sl + (uint32_t)grp * (8 * D) + lm_off);
#pragma unroll
        for (int g = 0; g < GH; ++g) r.s[g] = lds128(sl + s_off + g * (TOK * 2) + grp * 16);
    };
    uint4 low[GH];                                 // places of the low bytes of this lane's token of the stage's groups
    auto places = [&](uint32_t sl) {
#pragma unroll
        for (int g = 0; g < GH; ++g) low[g] = lds128(sl + low_off + g * (TOK * 2));
    };
    auto fetch_low = [&](Grp& r, int grp) {
#pragma unroll
        for (int g = 0; g < GH; ++g) {
            const uint32_t w = u4w(low[g], grp >> 1);
            ldm(r.l[g], lm_low + 2 * (grp & 1 ? w >> 16 : w & 0xFFFFu));
        }
    };
    uint32_t acc[GH];
    auto token = [&](const Grp& r, int u, bool with_low) {
        uint32_t k = 0;
        if (!with_low) k = __byte_perm(r.h[u >> 1], 0x80808080u, u & 1 ? 0x3424 : 0x1404);
#pragma unroll
        for (int g = 0; g < GH; ++g) {
            if (with_low) k = __byte_perm(r.h[u >> 1], r.l[g][u >> 1], u & 1 ? 0x3726 : 0x1504);
            acc[g] = v_fma(k, v_dup(u4w(r.s[g], u >> 1), u & 1), acc[g]);
        }
    };
    if (p.early) pdl_wait();
    bool alive = true;
    int slot = 0;
    uint32_t parity = 0;
    const int nsf = n / TOK, rest = n - nsf * TOK;
#pragma unroll 1
    for (int unit = first_unit; unit < p.units; unit += stride) {
#pragma unroll
        for (int g = 0; g < GH; ++g) acc[g] = 0;
        Grp r[NB];
        uint32_t sl = ring + (uint32_t)slot * SLOT, any = 0;
        if (alive && nst > 0) {
            alive = mbar_wait(bar_full + slot * 8, parity);
            any = lds32(sl + OFF_ANY);
#pragma unroll
            for (int j = 0; j < NB; ++j) fetch(r[j], sl, j);
        }
        // One full stage per iteration, straight-line; on entry r holds the bytes of its first NB groups.
#pragma unroll 1
        for (int left = nsf; left > 0 && alive; --left) {
            const int cslot = slot;
            if (++slot == nf) { slot = 0; parity ^= 1u; }
            const uint32_t nsl = ring + (uint32_t)slot * SLOT, nbar = bar_full + slot * 8;
            const bool more = left > 1 || rest > 0;
            uint32_t nany = 0;
            auto stage = [&](auto with_low) {
                constexpr bool LOW = decltype(with_low)::value;
#pragma unroll
                for (int j = 0; j < NG; ++j) {
                    if (j + NB == NG) {
                        // the next stage (when there is none: stale bytes, unused)
                        if (more) alive = mbar_wait(nbar, parity);
                        nany = lds32(nsl + OFF_ANY);
                    }
#pragma unroll
                    for (int u = 0; u < 8; ++u) token(r[j % NB], u, LOW);
                    if (j + NB < NG) {
                        fetch(r[j % NB], sl, j + NB);
                        if (LOW) fetch_low(r[j % NB], j + NB);
                    } else {
                        fetch(r[j % NB], nsl, j + NB - NG);
                    }
                }
            };
            if (__builtin_expect(any == 0, 1)) {
                stage(std::false_type{});
            } else {
                places(sl);
#pragma unroll
                for (int j = 0; j < NB; ++j) fetch_low(r[j], j);
                stage(std::true_type{});
            }
            // the stage is consumed: hand back its ring slot
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_free + cslot * 8);
            sl = nsl;
            any = nany;
        }
        if (rest > 0) {
            // last, partial stage (rows beyond the last token hold stale bytes: not accumulated)
            if (alive) {
                if (any != 0) places(sl);
#pragma unroll
                for (int k = 0; k < NG; ++k) {
                    if (8 * k >= rest) break;
                    fetch(r[0], sl, k);
                    if (any != 0) {
                        fetch_low(r[0], k);
                    } else {
#pragma unroll
                        for (int g = 0; g < GH; ++g)
#pragma unroll
                            for (int e = 0; e < 4; ++e) r[0].l[g][e] = 0x80808080u;
                    }
#pragma unroll
                    for (int u = 0; u < 8; ++u)
                        if (8 * k + u < rest) token(r[0], u, true);
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_free + slot * 8);
            if (++slot == nf) { slot = 0; parity ^= 1u; }
        }
#pragma unroll
        for (int g = 0; g < GH; ++g) {
            const size_t at = ((size_t)unit * NH + h0 + g) * 64 + pair;
            if (p.res) {
                const uint32_t t = reinterpret_cast<const uint32_t*>(p.res)[at];
                const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&acc[g]));
                const float2 b = __half22float2(*reinterpret_cast<const __half2*>(&t));
                const __half2 c = __floats2half2_rn(a.x + b.x, a.y + b.y);
                acc[g] = *reinterpret_cast<const uint32_t*>(&c);
            }
            reinterpret_cast<uint32_t*>(p.o)[at] = alive ? acc[g] : 0x7E007E00u;
        }
    }
}

}  // namespace akv

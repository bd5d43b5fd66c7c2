// A prompt (or its next chunk) through an attention layer, bf16: RoPE of q and k with the rows appended to the caches, and
// causal attention over everything cached so far on the 5th-generation tensor cores.
// (reference: check_and_apply_qk_rope, modify_llama.py:68-80; the dense attention of a prompt, spotlight_generation.py:145-147,217-224.)
//
// Attention: one CTA per (batch row, kv head, 256 query rows). The G query heads of a kv head share its K and V, so a
// tile's 128 rows are (token, head of the group) pairs, tokens slowest: 128 / G consecutive tokens (a group size that does
// not divide 128 leaves the last rows of a tile unused). Two tiles per CTA, so that the tensor core works on one while the
// softmax of the other runs. TMEM: S0 | S1 | O0 | O1, 128 fp32 columns each; P (bf16 pairs) takes the first half of its S.
//   producer  K and V tiles of 128 keys by TMA (no multicast), four 32 KB slots   -> kv_full[slot]
//   issuer    S_t = Q_t K^T (8 x M128 N128 K16, both operands in shared memory)   -> s_full[t]
//             O_t += P_t V  (8 x M128 N128 K16, P in TMEM, V rows as they lie in the cache: an MN-major operand)
//   softmax   4 warps per tile, a thread per row (no shuffles): online softmax in the exp2 domain, fp32; the running
//             maximum moves only when a row's grew by more than 2^8 (then O is rescaled in TMEM): sums stay exact to fp32
//             either way, as the factor cancels in O / l                            -> p_full[t]
// The tensor pipe executes in issue order, so S_t(j+1), issued behind O_t += P_t(j) V, is also the signal that the latter is
// over. What bounds it: a tile's chain P -> O += P V -> next S (TMEM has no room for a second S beside two O). The exponentials
// (16 a clock and SM: 1024 clocks per 128 x 128 tile) and the tensor core (two contractions of 512) are each about half
// busy; letting the two tiles' exponentials take turns changes nothing (136.4 us against 137).
// Blocks are ordered longest first (the last rows of a prompt see the most keys), so the tail of the launch is short.
// Measured (32 / 8 heads): 131 us for a prompt of 4001 tokens, 1.00 PFLOP/s of causal work, where torch's attention under the
// same mask took 3 406 us. The grid does not split the keys, so a short chunk over a long context fills few SMs (64 tokens: 8 CTAs); it
// is still the shorter way (whole layer call, torch's path in brackets): 2 tokens over 32 000 keys 487 us (983), 64 over 32 000
// 489 (991), 512 over 32 000 501 (1 010), 64 over 4 096 78 (189), 28 / 4 heads 64 over 120 000 1 780 (3 430).
// Error against 64 bits: 1.00 of torch's over prompts of 64 to 4096 tokens with up to 700 keys before them, at most 1.04 where torch takes
// its kernel with the exact maximum (1.20 with scores of deviation 4).
// Every wait is bounded; one that runs out raises sl_hash_status, the CTA lets its copies land, frees its TMEM and returns.
#include "sl_common.cuh"
#include "sl_tc.cuh"

namespace {

using namespace sltc;

constexpr int PF_THREADS = 10 * 32;                  // softmax of tile 0, of tile 1, producer, issuer
constexpr int PF_SLOTS = 4;
constexpr unsigned PF_TILE = 128 * 128 * 2, PF_SLAB = PF_TILE / 2;      // 128 rows: two slabs of 64 columns, rows of 128 bytes
constexpr unsigned PF_OFF_KV = 2 * PF_TILE, PF_OFF_BAR = PF_OFF_KV + PF_SLOTS * PF_TILE, PF_OFF_MISC = PF_OFF_BAR + 16 * 8,
                   PF_SMEM = PF_OFF_MISC + 16 + 1024;
constexpr float PF_SCALE = 0.08838834764831845f * 1.4426950408889634f;  // 1/sqrt(128) in the exp2 domain

struct PrefillArgs {
    int B, KH, G, tpt;                    // tpt: tokens per tile of 128 rows
    long long T, pos0;                    // new tokens, tokens before them
    long long nqb;                        // query blocks (of 2 * tpt tokens) per (batch row, kv head)
    __nv_bfloat16* out;                   // [B,T,KH*G,128]
    int* status;
};

__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// descriptor of a V tile: rows (keys, the contraction's K) of 128 bytes along N, 128-byte swizzle; groups of 8 keys are
// 1024 bytes apart, the second 64 columns one slab further
__device__ __forceinline__ unsigned long long smem_desc_mn(unsigned addr) {
    return (unsigned long long)((addr >> 4) & 0x3fffu) | ((unsigned long long)(PF_SLAB >> 4) << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}

__global__ void __launch_bounds__(PF_THREADS, 1)
prefill_attn_kernel(const __grid_constant__ CUtensorMap qmap, const __grid_constant__ CUtensorMap kmap,
                    const __grid_constant__ CUtensorMap vmap, const PrefillArgs a) {
    extern __shared__ unsigned char smem_raw[];
    const unsigned raw = (unsigned)__cvta_generic_to_shared(smem_raw);
    const unsigned base = (raw + 1023u) & ~1023u;
    unsigned char* gsm = smem_raw + (base - raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    volatile int* abort_flag = reinterpret_cast<volatile int*>(gsm + PF_OFF_MISC + 4);
    unsigned* tmem_slot = reinterpret_cast<unsigned*>(gsm + PF_OFF_MISC);
    auto bar = [&](int i) { return base + PF_OFF_BAR + (unsigned)i * 8u; };
    constexpr int Q_FULL = 0, KV_FULL = 1 /* .. 4 */, KV_FREE = 5 /* .. 8 */, S_FULL = 9 /* , 10 */, P_FULL = 11 /* , 12 */, O_FULL = 13;

    if (tid == 0) {
        *abort_flag = 0;
        mbar_init(bar(Q_FULL), 1); mbar_init(bar(O_FULL), 1);
        for (int i = 0; i < PF_SLOTS; ++i) { mbar_init(bar(KV_FULL + i), 1); mbar_init(bar(KV_FREE + i), 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(bar(S_FULL + i), 1); mbar_init(bar(P_FULL + i), 128); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 9) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(base + PF_OFF_MISC) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = *tmem_slot;

    const int bhn = a.B * a.KH;
    const long long qb = a.nqb - 1 - (long long)blockIdx.x / bhn;
    const int bh = (int)(blockIdx.x % bhn), b = bh / a.KH, h = bh - b * a.KH;
    const long long tok0 = qb * 2 * a.tpt;                                   // first token of the block
    const long long last = a.pos0 + min(a.T, tok0 + 2 * a.tpt) - 1;          // last key any of its rows sees
    const int nkv = (int)(last / 128) + 1;
    bool failed = false;

    if (warp < 8) {
        // ================= softmax: thread = row = TMEM lane =================
        const int t = warp >> 2, row = (warp & 3) * 32 + lane;
        const unsigned t_row = tmem + ((unsigned)((warp & 3) * 32) << 16), t_s = t_row + 128u * t, t_o = t_row + 256u + 128u * t;
        const long long first = tok0 + (long long)t * a.tpt;                 // first token of the tile
        const int rt = row / a.G, rg = row - rt * a.G;
        const long long limit = a.pos0 + first + rt;                         // last key this row sees
        const long long open = a.pos0 + first;                               // every row of the tile sees the keys up to here
        float m = -INFINITY, l = 0.0f;
        for (int j = 0; j < nkv; ++j) {
            if (!__all_sync(0xffffffffu, mbar_wait(bar(S_FULL + t), (unsigned)j & 1u, abort_flag))) { failed = true; break; }
            tc_fence_after();
            float s[4][32];
#pragma unroll
            for (int c = 0; c < 4; ++c) tmem_ld32(t_s + 32u * c, reinterpret_cast<unsigned (&)[32]>(s[c]));
            tmem_wait_ld();
            if ((long long)j * 128 + 127 > open) {
                const int keep = (int)min(limit - (long long)j * 128, 128ll);  // columns up to this one (may be negative: none)
#pragma unroll
                for (int c = 0; c < 4; ++c)
#pragma unroll
                    for (int e = 0; e < 32; ++e)
                        if (32 * c + e > keep) s[c][e] = -INFINITY;
            }
            float mx[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                mx[c] = s[c][0];
#pragma unroll
                for (int e = 1; e < 32; ++e) mx[c] = fmaxf(mx[c], s[c][e]);
            }
            const float mn = fmaxf(m, fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])));
            if (j == 0) {
                m = mn;
            } else if (__any_sync(0xffffffffu, (mn - m) * PF_SCALE > 8.0f)) {
                const float f = mn == -INFINITY ? 1.0f : ex2((m - mn) * PF_SCALE);     // O += P V of the tile before is over (see above)
                m = mn;
                l *= f;
#pragma unroll 1
                for (int c = 0; c < 8; ++c) {
                    unsigned o[16];
                    tmem_ld16(t_o + 16u * c, o);
                    tmem_wait_ld();
#pragma unroll
                    for (int e = 0; e < 16; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * f);
                    tmem_st16(t_o + 16u * c, o);
                }
            }
            const float ms = m == -INFINITY ? 0.0f : m * PF_SCALE;
            float sum[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                unsigned pk[16];
#pragma unroll
                for (int e = 0; e < 16; ++e) {
                    const float p0 = ex2(fmaf(s[c][2 * e], PF_SCALE, -ms)), p1 = ex2(fmaf(s[c][2 * e + 1], PF_SCALE, -ms));
                    sum[(2 * e) & 3] += p0;
                    sum[(2 * e + 1) & 3] += p1;
                    pk[e] = pack2(p0, p1);
                }
                tmem_st16(t_s + 16u * c, pk);
            }
            l += (sum[0] + sum[1]) + (sum[2] + sum[3]);
            tmem_wait_st();
            tc_fence_before();
            mbar_arrive(bar(P_FULL + t));
        }
        if (!failed && !__all_sync(0xffffffffu, mbar_wait(bar(O_FULL), 0u, abort_flag))) failed = true;
        if (!failed) {
            tc_fence_after();
            const bool store = rt < a.tpt && first + rt < a.T;
            const float inv = 1.0f / l;
            __nv_bfloat16* dst = a.out + (((long long)b * a.T + first + rt) * a.KH * a.G + (long long)h * a.G + rg) * 128;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                unsigned o[32];
                tmem_ld32(t_o + 32u * c, o);
                tmem_wait_ld();
                if (store) {
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        uint4 w;
                        w.x = pack2(__uint_as_float(o[8 * e]) * inv, __uint_as_float(o[8 * e + 1]) * inv);
                        w.y = pack2(__uint_as_float(o[8 * e + 2]) * inv, __uint_as_float(o[8 * e + 3]) * inv);
                        w.z = pack2(__uint_as_float(o[8 * e + 4]) * inv, __uint_as_float(o[8 * e + 5]) * inv);
                        w.w = pack2(__uint_as_float(o[8 * e + 6]) * inv, __uint_as_float(o[8 * e + 7]) * inv);
                        *reinterpret_cast<uint4*>(dst + 32 * c + 8 * e) = w;
                    }
                }
            }
        }
    } else if (warp == 8 && lane == 0) {
        // ================= producer =================
        const unsigned rows = (unsigned)(a.tpt * a.G);
        mbar_expect_tx(bar(Q_FULL), 2u * rows * 256u);
        for (int t = 0; t < 2; ++t)                                          // a tile past the end reads zeros
            for (int c = 0; c < 2; ++c)
                tma_load_4d(base + t * PF_TILE + c * PF_SLAB, &qmap, bar(Q_FULL), 64 * c, h * a.G, (int)(tok0 + t * a.tpt), b);
        const int n = 2 * nkv;
        int i = 0;
        for (; i < n; ++i) {
            const int slot = i % PF_SLOTS;
            if (i >= PF_SLOTS && !mbar_wait(bar(KV_FREE + slot), (unsigned)(i / PF_SLOTS - 1) & 1u, abort_flag)) { failed = true; break; }
            const unsigned dst = base + PF_OFF_KV + slot * PF_TILE;
            const CUtensorMap* map = (i & 1) ? &vmap : &kmap;
            mbar_expect_tx(bar(KV_FULL + slot), PF_TILE);
            tma_load_4d(dst, map, bar(KV_FULL + slot), 0, (i >> 1) * 128, h, b);
            tma_load_4d(dst + PF_SLAB, map, bar(KV_FULL + slot), 64, (i >> 1) * 128, h, b);
        }
        // the CTA's memory must not go before its copies have landed: they all have where the issuer got to its end, else wait here
        for (int s = 0; s < PF_SLOTS && s < i; ++s) {
            const int lasti = s + (i - 1 - s) / PF_SLOTS * PF_SLOTS;
            for (unsigned k = 0; k < WAIT_LIMIT && !mbar_test(bar(KV_FULL + s), (unsigned)(lasti / PF_SLOTS) & 1u); ++k) __nanosleep(256);
        }
        for (unsigned k = 0; k < WAIT_LIMIT && !mbar_test(bar(Q_FULL), 0u); ++k) __nanosleep(256);
    } else if (warp == 9 && lane == 0) {
        // ================= issuer =================
        constexpr unsigned IS = instr_desc(128), IO = instr_desc(128) | (1u << 16);      // the second: B (V) is MN-major
        auto scores = [&](int t, unsigned kslot) {
#pragma unroll
            for (int ks = 0; ks < 8; ++ks) {
                const unsigned o = (unsigned)(ks >> 2) * PF_SLAB + (unsigned)(ks & 3) * 32u;
                mma_ss(tmem + 128u * t, smem_desc(base + t * PF_TILE + o), smem_desc(base + PF_OFF_KV + kslot * PF_TILE + o), IS, ks > 0 ? 1u : 0u);
            }
            tc_commit(bar(S_FULL + t));
        };
        if (!mbar_wait(bar(Q_FULL), 0u, abort_flag) || !mbar_wait(bar(KV_FULL), 0u, abort_flag)) failed = true;
        if (!failed) {
            tc_fence_after();
            scores(0, 0);
            scores(1, 0);
            tc_commit(bar(KV_FREE));
        }
        for (int j = 0; j < nkv && !failed; ++j) {
            const int iv = 2 * j + 1, ik = 2 * j + 2;
            const unsigned vslot = iv % PF_SLOTS, kslot = ik % PF_SLOTS;
            if (!mbar_wait(bar(KV_FULL + vslot), (unsigned)(iv / PF_SLOTS) & 1u, abort_flag)) { failed = true; break; }
            if (j + 1 < nkv && !mbar_wait(bar(KV_FULL + kslot), (unsigned)(ik / PF_SLOTS) & 1u, abort_flag)) { failed = true; break; }
            for (int t = 0; t < 2; ++t) {
                if (!mbar_wait(bar(P_FULL + t), (unsigned)j & 1u, abort_flag)) { failed = true; break; }
                tc_fence_after();
#pragma unroll
                for (int ks = 0; ks < 8; ++ks)
                    mma_ts(tmem + 256u + 128u * t, tmem + 128u * t + 8u * ks, smem_desc_mn(base + PF_OFF_KV + vslot * PF_TILE + ks * 2048u), IO,
                           (j | ks) ? 1u : 0u);
                if (j + 1 < nkv) scores(t, kslot);
            }
            if (failed) break;
            tc_commit(bar(KV_FREE + vslot));
            if (j + 1 < nkv) tc_commit(bar(KV_FREE + kslot));
        }
        if (!failed) tc_commit(bar(O_FULL));
    }
    if (failed) {
        *abort_flag = 1;
        if (a.status) *reinterpret_cast<volatile int*>(a.status) = 3;
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 9) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
}

// ---- RoPE of q and k and the append of K and V rows, one pass: a thread rotates 8 dimensions of the first half of a row with
// the 8 of the second half they pair with. torch's rounding points (x * cos -> bf16, rotate_half(x) * sin -> bf16, sum
// -> bf16). Bound by its bytes: 98 MB for 4001 tokens of 32 + 2 x 8 heads, 18 us (torch's operators: 350 us).
struct RopeArgs {
    const __nv_bfloat16* q; const __nv_bfloat16* k; const __nv_bfloat16* v;      // [B,T,heads,128]
    const __nv_bfloat16* cos; const __nv_bfloat16* sin;                          // [T,128]
    __nv_bfloat16* q_rot; __nv_bfloat16* kc; __nv_bfloat16* vc;                  // caches at the first new row
    long long kv_b, kv_tok, kv_h;
    long long T; int QH, KH;
    long long rows;                                                              // B * T
};

__global__ void __launch_bounds__(256) rope_append_kernel(const RopeArgs a) {
    const int heads = a.QH + 2 * a.KH;
    const long long total = a.rows * heads * 8;
    for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < total; i += (long long)gridDim.x * 256) {
        const int c = (int)(i & 7) * 8;                                          // dimensions c.. and 64 + c..
        const long long rh = i >> 3;
        const long long r = rh / heads;
        const int head = (int)(rh - r * heads);
        const long long b = r / a.T, t = r - b * a.T;
        const __nv_bfloat16* src;
        __nv_bfloat16* dst;
        if (head < a.QH) {
            src = a.q + (r * a.QH + head) * 128;
            dst = a.q_rot + (r * a.QH + head) * 128;
        } else {
            const int hk = head - a.QH < a.KH ? head - a.QH : head - a.QH - a.KH;
            const long long o = b * a.kv_b + t * a.kv_tok + hk * a.kv_h;
            src = (head < a.QH + a.KH ? a.k : a.v) + (r * a.KH + hk) * 128;
            dst = (head < a.QH + a.KH ? a.kc : a.vc) + o;
        }
        uint4 lo = sl::ld_stream_v4(reinterpret_cast<const uint4*>(src + c)), hi = sl::ld_stream_v4(reinterpret_cast<const uint4*>(src + 64 + c));
        if (head < a.QH + a.KH) {
            const uint4 cl = __ldg(reinterpret_cast<const uint4*>(a.cos + t * 128 + c)), ch = __ldg(reinterpret_cast<const uint4*>(a.cos + t * 128 + 64 + c));
            const uint4 sn = __ldg(reinterpret_cast<const uint4*>(a.sin + t * 128 + c)), sh = __ldg(reinterpret_cast<const uint4*>(a.sin + t * 128 + 64 + c));
            unsigned* L = reinterpret_cast<unsigned*>(&lo);
            unsigned* H = reinterpret_cast<unsigned*>(&hi);
            auto part = [](unsigned x, unsigned cs, unsigned y, unsigned sn2, float sign) {      // x cos + sign * y sin, a pair
                const float x0 = __uint_as_float(x << 16), x1 = __uint_as_float(x & 0xffff0000u);
                const float c0 = __uint_as_float(cs << 16), c1 = __uint_as_float(cs & 0xffff0000u);
                const float y0 = sign * __uint_as_float(y << 16), y1 = sign * __uint_as_float(y & 0xffff0000u);
                const float s0 = __uint_as_float(sn2 << 16), s1 = __uint_as_float(sn2 & 0xffff0000u);
                const unsigned p = pack2(x0 * c0, x1 * c1), q = pack2(y0 * s0, y1 * s1);
                return pack2(__uint_as_float(p << 16) + __uint_as_float(q << 16), __uint_as_float(p & 0xffff0000u) + __uint_as_float(q & 0xffff0000u));
            };
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const unsigned x = L[e], y = H[e];
                L[e] = part(x, reinterpret_cast<const unsigned*>(&cl)[e], y, reinterpret_cast<const unsigned*>(&sn)[e], -1.0f);
                H[e] = part(y, reinterpret_cast<const unsigned*>(&ch)[e], x, reinterpret_cast<const unsigned*>(&sh)[e], 1.0f);
            }
        }
        *reinterpret_cast<uint4*>(dst + c) = lo;
        *reinterpret_cast<uint4*>(dst + 64 + c) = hi;
    }
}

}  // namespace

extern "C" int sl_rope_append(const void* d_q, const void* d_k, const void* d_v, int dtype, int B, int64_t T, int QH, int KH,
                              const void* d_cos, const void* d_sin, void* d_q_rot, void* d_k_cache, void* d_v_cache,
                              const sl_kv_layout* kv, int64_t pos, void* stream) {
    SL_REQUIRE(d_q && d_k && d_v && d_cos && d_sin && d_q_rot && d_k_cache && d_v_cache && kv, SL_EINVAL, "sl_rope_append: null pointer");
    SL_REQUIRE(dtype == SL_BF16, SL_EINVAL, "sl_rope_append: dtype %d (bf16 only)", dtype);
    SL_REQUIRE(B > 0 && T >= 0 && QH > 0 && KH > 0 && pos >= 0, SL_ESHAPE, "sl_rope_append: bad shape");
    SL_REQUIRE(kv->token_stride >= 128 && kv->head_stride >= 128 && kv->batch_stride >= 0 && kv->token_stride % 8 == 0 &&
               kv->head_stride % 8 == 0 && kv->batch_stride % 8 == 0, SL_EALIGN, "sl_rope_append: cache strides");
    for (const void* p : {d_q, d_k, d_v, d_cos, d_sin, (const void*)d_q_rot, (const void*)d_k_cache, (const void*)d_v_cache})
        SL_REQUIRE(sl::aligned16(p), SL_EALIGN, "sl_rope_append: pointer not 16-byte aligned");
    if (T == 0) return SL_OK;
    RopeArgs a = {};
    a.q = (const __nv_bfloat16*)d_q; a.k = (const __nv_bfloat16*)d_k; a.v = (const __nv_bfloat16*)d_v;
    a.cos = (const __nv_bfloat16*)d_cos; a.sin = (const __nv_bfloat16*)d_sin;
    a.q_rot = (__nv_bfloat16*)d_q_rot;
    a.kc = (__nv_bfloat16*)d_k_cache + pos * kv->token_stride;
    a.vc = (__nv_bfloat16*)d_v_cache + pos * kv->token_stride;
    a.kv_b = kv->batch_stride; a.kv_tok = kv->token_stride; a.kv_h = kv->head_stride;
    a.T = T; a.QH = QH; a.KH = KH; a.rows = (long long)B * T;
    const long long blocks = std::min<long long>((a.rows * (QH + 2 * KH) * 8 + 255) / 256, (long long)sl::sm_count() * 32);
    rope_append_kernel<<<(unsigned)blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(a);
    SL_CUDA_OK(cudaGetLastError());
    return SL_OK;
}

extern "C" int sl_prefill_attn(const void* d_q, const void* d_k_cache, const void* d_v_cache, int dtype, const sl_kv_layout* kv, int B,
                               int64_t T, int QH, int KH, int64_t pos, void* d_out, void* stream) {
    SL_REQUIRE(d_q && d_k_cache && d_v_cache && kv && d_out, SL_EINVAL, "sl_prefill_attn: null pointer");
    SL_REQUIRE(dtype == SL_BF16, SL_EINVAL, "sl_prefill_attn: dtype %d (bf16 only)", dtype);
    SL_REQUIRE(B > 0 && T >= 0 && QH > 0 && KH > 0 && QH % KH == 0 && QH / KH <= 128 && pos >= 0, SL_ESHAPE, "sl_prefill_attn: bad shape");
    SL_REQUIRE(pos + T <= 0x7fffff00ll && B <= 65535 && KH <= 65535, SL_ESHAPE, "sl_prefill_attn: shape too large");
    SL_REQUIRE(sl::aligned16(d_q) && sl::aligned16(d_k_cache) && sl::aligned16(d_v_cache) && sl::aligned16(d_out), SL_EALIGN,
               "sl_prefill_attn: pointer not 16-byte aligned");
    SL_REQUIRE(kv->token_stride >= 128 && kv->head_stride >= 128 && kv->token_stride % 8 == 0 && kv->head_stride % 8 == 0 &&
               (B == 1 || (kv->batch_stride > 0 && kv->batch_stride % 8 == 0)), SL_EALIGN, "sl_prefill_attn: cache strides");
    if (T == 0) return SL_OK;
    EncodeTiledFn enc = encode_fn();
    SL_REQUIRE(enc, SL_ECUDA, "sl_prefill_attn: cuTensorMapEncodeTiled not available");
    const int G = QH / KH, tpt = 128 / G;
    const long long n = pos + T;
    CUtensorMap qm, km, vm;
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    {
        const cuuint64_t dim[4] = {128, (cuuint64_t)QH, (cuuint64_t)T, (cuuint64_t)B};
        const cuuint64_t str[3] = {256, (cuuint64_t)QH * 256, (cuuint64_t)T * QH * 256};
        const cuuint32_t box[4] = {64, (cuuint32_t)G, (cuuint32_t)tpt, 1};
        SL_REQUIRE(enc(&qm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(d_q), dim, str, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                       CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS,
                   SL_EINVAL, "sl_prefill_attn: tensor map of q");
    }
    for (int i = 0; i < 2; ++i) {
        // the token extent ends at the last cached row: keys past it read zeros, whatever the cache holds there
        const cuuint64_t dim[4] = {128, (cuuint64_t)n, (cuuint64_t)KH, (cuuint64_t)B};
        const cuuint64_t str[3] = {(cuuint64_t)kv->token_stride * 2, (cuuint64_t)kv->head_stride * 2,
                                   (cuuint64_t)(B > 1 ? kv->batch_stride : n * kv->token_stride) * 2};
        const cuuint32_t box[4] = {64, 128, 1, 1};
        SL_REQUIRE(enc(i ? &vm : &km, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(i ? d_v_cache : d_k_cache), dim, str, box, estr,
                       CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                       CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS,
                   SL_EINVAL, "sl_prefill_attn: tensor map of the cache");
    }
    PrefillArgs a = {};
    a.B = B; a.KH = KH; a.G = G; a.tpt = tpt; a.T = T; a.pos0 = pos;
    a.nqb = (T + 2 * tpt - 1) / (2 * tpt);
    a.out = (__nv_bfloat16*)d_out;
    a.status = sl::tc_status_word();
    const long long blocks = a.nqb * B * KH;
    SL_REQUIRE(blocks <= 0x7fffffffll, SL_ESHAPE, "sl_prefill_attn: too many blocks");
    SL_CUDA_OK(cudaFuncSetAttribute(prefill_attn_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PF_SMEM));
    prefill_attn_kernel<<<(unsigned)blocks, PF_THREADS, PF_SMEM, static_cast<cudaStream_t>(stream)>>>(qm, km, vm, a);
    SL_CUDA_OK(cudaGetLastError());
    return SL_OK;
}

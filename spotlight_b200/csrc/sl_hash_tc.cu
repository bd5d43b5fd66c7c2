// Code-cache build at prefill on the 5th-generation tensor cores: hash MLP 128 -> {256, 128} -> 128 (the narrow one also
// in the reference's residual form) and linear hash 128 -> 128 (bf16),
// sign and pack of many rows of one head per CTA. This is the one dense contraction of the retrieval path
// (reference math: spotlight/modifiers/spotlight_generation.py:229-255).
//
// One persistent CTA per SM works on 128-row tiles of one head, one tile after the other. The head's weights stay in shared memory
// for the whole launch, transposed to K-major rows in the 128-byte-swizzled layout tcgen05.mma reads; the
// accumulators live in tensor memory (TMEM); input tiles arrive by TMA (cp.async.bulk.tensor, one CTA per copy,
// this GPU's own memory) straight into the same swizzled layout.
//
// The MLP kernel keeps TWO tiles in flight, each with 256 columns of TMEM, an input stage, eight epilogue warps and an
// issuing thread of its own, so that one tile's contractions run under the other's activations (the epilogues take
// turns). TMEM of a tile: layer 1 in [0,D1); a warp reads the columns 64 w .. (of every 128) of its rows and writes the packed
// hidden values back over [64 w, +64), columns it has read itself; layer 2's result in [128,256).
//   TMA   X tile [128 x 128]                                   -> x_full
//   MMA1  D1[128 x D1] = X W1             (8 x  M128 N=D1 K16)  -> d1_full (the input stage takes the next rows; in the
//         residual form after h_full, as the epilogue adds the rows)
//   EPI1  D1 -> registers, torch's rounding points (matmul -> bf16, + bias -> bf16, SiLU -> bf16, + input -> bf16 in the
//         residual form), packed pairs of bf16 written to H: the A operand of layer 2     -> h_full
//   MMA2  D2[128 x 128] = H W2            (D1/16 x M128 N128 K16, A from TMEM) -> d2_full
//   EPI2  D2 -> registers, rounding points, sign bit of every value: a thread holds two 32-bit words of its
//         row's code and stores them                            -> d2_free
// Bound by the activation: two MUFU operations per hidden value, 4096 clocks per tile of 128 x 256, against 2048 of the tensor
// core. 128 -> 256 -> 128, 131 072 x 8 rows, contiguous or the K half of a fused cache: 171 us back to back (267 with one tile in
// flight and a table of SiLU values in shared memory); 128 -> 128 -> 128 residual: 136 us (231). The linear hash has a kernel of its own further
// down (one contraction per tile, bound by the stream of its input rows). With LOAD the input rows are new rows of a cache: the
// K rows leave for it from the input stage, the V rows are copied beside them, all by TMA, and the cache is
// not read back: 131 072 x 8 rows into a fused cache with their codes in 235 us, where two strided copies and the codes took 867.
// Every wait on an mbarrier is bounded; a wait that runs out raises the library's hash status word, the CTA lets its
// copies in flight land, frees its TMEM and returns.
// Same arithmetic as the warp-level kernel in sl_hash_mma.cu up to the order of the fp32 additions.
#include <mutex>

#include "sl_common.cuh"
#include "sl_tc.cuh"

namespace {

using namespace sltc;

constexpr int TC_EPI_WARPS = 16;                // two tiles x 4 lane quadrants x 2 column halves
constexpr int TC_THREADS = (TC_EPI_WARPS + 3) * 32;   // + an issuing warp per tile and one that copies V rows
constexpr int TC_TILE = 128;
constexpr unsigned X_BYTES = TC_TILE * 128 * 2, X_SLAB = X_BYTES / 2;

constexpr int VS = 4;                             // pieces of the V copy in flight
constexpr unsigned V_PIECE = 32 * 256;            // 32 whole rows

// shared memory of the MLP kernel, bytes from a 1024-byte boundary
template <int D1>
struct TcSmem {
    static constexpr unsigned W1 = 0, W2 = 128 * D1 * 2, X = 2 * W2, V = X + 2 * X_BYTES, B1 = V + VS * V_PIECE, B2 = B1 + D1 * 2, BAR = B2 + 256,
                              MISC = BAR + (12 + VS) * 8, BYTES = MISC + 16 + 1024;
};

struct HashTcArgs {
    long long T; int H; int B;
    const __nv_bfloat16* w1; const __nv_bfloat16* w2; const __nv_bfloat16* b1; const __nv_bfloat16* b2;
    uint32_t* codes; long long cs_b;
    long long tiles_per_b, n_tiles;
    int* status;                                  // mapped host word: 3 = a wait ran out
};

// sum of two pairs of bf16, each rounded to nearest even once: equal to the fp32 sum rounded to bf16
__device__ __forceinline__ unsigned add_bf16x2(unsigned x, unsigned y) {
    unsigned r;
    asm("add.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(x), "r"(y));
    return r;
}

// SiLU of a pair of bf16 at torch's rounding point: fp32 x / (1 + exp(-x)), rounded once. Computed as (x/4) * (1 / ((1 + 2^(-x log2 e)) / 4))
// with the approximate exponential and reciprocal (the quarter keeps the reciprocal of 1 + e^88 out of the denormals,
// which those flush): over all finite bf16 arguments the rounded result is the one of the accurate formula, bit for bit (tested
// exhaustively). Two MUFU operations per value; a table of the values in shared memory costs as many clocks (three-way bank
// conflicts), the index arithmetic and 16 KB that the copy of V rows needs.
__device__ __forceinline__ unsigned long long pair64(float lo, float hi) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ unsigned silu_pair(unsigned y) {
    const float NL = -1.4426950408889634f;
    const unsigned long long x = pair64(__uint_as_float(y << 16), __uint_as_float(y & 0xffff0000u));
    unsigned long long e, d, r, q;
    float t0, t1, r0, r1;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(e) : "l"(x), "l"(pair64(NL, NL)));
    asm("{\n\t.reg .f32 a, b;\n\tmov.b64 {a, b}, %2;\n\tex2.approx.ftz.f32 %0, a;\n\tex2.approx.ftz.f32 %1, b;\n\t}" : "=f"(t0), "=f"(t1) : "l"(e));
    asm("fma.rn.f32x2 %0, %1, %2, %2;" : "=l"(d) : "l"(pair64(t0, t1)), "l"(pair64(0.25f, 0.25f)));
    asm("{\n\t.reg .f32 a, b;\n\tmov.b64 {a, b}, %2;\n\trcp.approx.ftz.f32 %0, a;\n\trcp.approx.ftz.f32 %1, b;\n\t}" : "=f"(r0), "=f"(r1) : "l"(d));
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(q) : "l"(x), "l"(pair64(0.25f, 0.25f)));
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(q), "l"(pair64(r0, r1)));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r0), "=f"(r1) : "l"(r));
    return pack2(r0, r1);
}

// byte offset of element (row, k) of a K-major operand: slabs of 64 k, rows of 128 bytes, 16-byte chunks XORed with row % 8
__device__ __forceinline__ unsigned kmajor_off(int row, int k, int rows) {
    return (unsigned)((k >> 6) * rows * 128 + row * 128 + ((((k & 63) >> 3) ^ (row & 7)) << 4) + (k & 7) * 2);
}

// LOAD: one thread copies the V rows of the CTA's tiles by TMA, a quarter of a tile (32 whole rows) at a time, VS in
// flight, one barrier each. False when a bounded wait ran out (its copies have landed all the same).
__device__ __forceinline__ bool copy_v_rows(unsigned smem, unsigned bars, const CUtensorMap& vsrc, const CUtensorMap& vdst, const HashTcArgs& a,
                                            long long first, long long step, int h, volatile int* abort_flag) {
    const long long n = first < a.n_tiles ? 4 * ((a.n_tiles - 1 - first) / step + 1) : 0;
    auto place = [&](long long i, int& t0, int& b) {
        const long long tile = first + (i >> 2) * step, bb = tile / a.tiles_per_b;
        b = (int)bb; t0 = (int)((tile - bb * a.tiles_per_b) * TC_TILE) + (int)(i & 3) * 32;
    };
    auto load = [&](long long i) {
        const unsigned st = (unsigned)(i % VS);
        int t0, b;
        place(i, t0, b);
        mbar_expect_tx(bars + 8u * st, V_PIECE);
        tma_load_4d(smem + st * V_PIECE, &vsrc, bars + 8u * st, 0, t0, h, b);
    };
    long long loaded = 0, i = 0;
    for (; loaded < VS && loaded < n; ++loaded) load(loaded);
    bool ok = true;
    for (; i < n; ++i) {
        const unsigned st = (unsigned)(i % VS);
        if (!mbar_wait(bars + 8u * st, (unsigned)(i / VS) & 1u, abort_flag)) { ok = false; break; }
        int t0, b;
        place(i, t0, b);
        if (t0 < a.T) tma_store_4d(&vdst, smem + st * V_PIECE, 0, t0, h, b);
        bulk_commit();
        if (i >= 1 && loaded < n) { bulk_wait_read1(); load(loaded); ++loaded; }      // into the piece before this one, which has left
    }
    bulk_wait_read();
    for (; i < loaded; ++i)
        for (unsigned k = 0; k < WAIT_LIMIT && !mbar_test(bars + 8u * (unsigned)(i % VS), (unsigned)(i / VS) & 1u); ++k) __nanosleep(256);
    return ok;
}

// Sign bits of 16 pairs of bf16 as a code word: bit 2e <- low half > 0, bit 2e + 1 <- high half > 0 of pair e.
__device__ __forceinline__ unsigned signs16(const unsigned (&y)[16]) {
    unsigned w[2] = {0u, 0u};                 // eight pairs each: low halves in the even bits 0.., high halves in the even bits 16..
#pragma unroll
    for (int e = 0; e < 16; ++e) {
        __nv_bfloat162 v, z;
        reinterpret_cast<unsigned&>(v) = y[e];
        reinterpret_cast<unsigned&>(z) = 0u;
        w[e >> 3] |= __hgt2_mask(v, z) & (0x00010001u << (2 * (e & 7)));
    }
    return (w[0] & 0xffffu) | ((w[0] >> 16) << 1) | (w[1] << 16) | ((w[1] >> 16) << 17);
}

// D1: width of the hidden layer. RES (D1 == 128): the reference's residual form, layer output = f(x W + b) + input,
// rounded once more to bf16. LOAD: the input rows are new rows of a cache; the CTA stores every input tile from its
// stage to the K cache by TMA and copies the V rows of the same tile beside it.
template <int D1, bool RES, bool LOAD>
__global__ void __launch_bounds__(TC_THREADS, 1)
hash_encode_tc_kernel(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap kdst,
                      const __grid_constant__ CUtensorMap vsrc, const __grid_constant__ CUtensorMap vdst, const HashTcArgs a) {
    static_assert(D1 == 256 || (D1 == 128), "hidden width");
    static_assert(!RES || D1 == 128, "a residual layer keeps its width");
    using S = TcSmem<D1>;
    constexpr int NCH = D1 / 64;                              // 32-column pieces of D1 per epilogue warp
    extern __shared__ unsigned char smem_raw[];
    const unsigned raw = (unsigned)__cvta_generic_to_shared(smem_raw);
    const unsigned base = (raw + 1023u) & ~1023u;             // operand slabs start on 1024-byte boundaries
    unsigned char* g = smem_raw + (base - raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int h = blockIdx.y;
    volatile int* abort_flag = reinterpret_cast<volatile int*>(g + S::MISC + 4);
    unsigned* tmem_slot = reinterpret_cast<unsigned*>(g + S::MISC);
    auto bar = [&](int i) { return base + S::BAR + (unsigned)i * 8u; };
    constexpr int X_FULL = 0, D1_FULL = 2, H_FULL = 4, D2_FULL = 6, D2_FREE = 8 /* each + tile in flight */, TURN = 10, V_FULL = 12 /* .. */;

    // ---- set-up: barriers, TMEM, this head's weights (transposed to K-major) and biases
    if (tid == 0) {
        *abort_flag = 0;
        for (int p = 0; p < 2; ++p) {
            mbar_init(bar(X_FULL + p), 1); mbar_init(bar(D1_FULL + p), 1); mbar_init(bar(D2_FULL + p), 1);
            mbar_init(bar(H_FULL + p), TC_EPI_WARPS * 16); mbar_init(bar(D2_FREE + p), TC_EPI_WARPS * 16);
            mbar_init(bar(TURN + p), TC_EPI_WARPS * 16);
        }
        for (int i = 0; i < VS; ++i) mbar_init(bar(V_FULL + i), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == TC_EPI_WARPS) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(base + S::MISC) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    {
        // a warp takes 32 consecutive k of 8 columns: each lane reads 16 bytes of its row and writes 8 halfwords; the
        // 32 lanes of a store fall into distinct banks (k runs along the swizzled 128-byte row)
        const int NWARP = TC_THREADS / 32;
        constexpr int NG1 = D1 / 8;                                                               // groups of 8 n per row of W1
        const uint4* w1 = reinterpret_cast<const uint4*>(a.w1 + (long long)h * 128 * D1);         // [k][n]
        for (int task = warp; task < 4 * NG1; task += NWARP) {
            const int k = (task / NG1) * 32 + lane, n0 = (task % NG1) * 8;
            const uint4 v = w1[k * NG1 + (task % NG1)];
            const unsigned short* e = reinterpret_cast<const unsigned short*>(&v);
#pragma unroll
            for (int c = 0; c < 8; ++c) *reinterpret_cast<unsigned short*>(g + S::W1 + kmajor_off(n0 + c, k, D1)) = e[c];
        }
        const uint4* w2 = reinterpret_cast<const uint4*>(a.w2 + (long long)h * D1 * 128);         // [k][n], 16 groups of 8 n per row
        for (int task = warp; task < (D1 / 32) * 16; task += NWARP) {
            const int k = (task >> 4) * 32 + lane, n0 = (task & 15) * 8;
            const uint4 v = w2[k * 16 + (task & 15)];
            const unsigned short* e = reinterpret_cast<const unsigned short*>(&v);
#pragma unroll
            for (int c = 0; c < 8; ++c) *reinterpret_cast<unsigned short*>(g + S::W2 + kmajor_off(n0 + c, k, 128)) = e[c];
        }
        __nv_bfloat16* sb1 = reinterpret_cast<__nv_bfloat16*>(g + S::B1);
        __nv_bfloat16* sb2 = reinterpret_cast<__nv_bfloat16*>(g + S::B2);
        for (int i = tid; i < D1; i += TC_THREADS) sb1[i] = a.b1 ? a.b1[(long long)h * D1 + i] : __float2bfloat16_rn(0.0f);
        for (int i = tid; i < 128; i += TC_THREADS) sb2[i] = a.b2 ? a.b2[(long long)h * 128 + i] : __float2bfloat16_rn(0.0f);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");     // the weights were written by ordinary stores, the tensor core reads them
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = *tmem_slot;

    const long long first = blockIdx.x, step = gridDim.x;            // this CTA's tiles; tile in flight p takes every second one
    bool failed = false;

    if (warp < TC_EPI_WARPS) {
        // ================= epilogue warps: thread = row = TMEM lane and a half of the columns of tile in flight p =================
        const int p = warp >> 3, q = warp & 3, hw = (warp >> 2) & 1, row = q * 32 + lane;
        const unsigned t_row = tmem + ((unsigned)(q * 32) << 16) + 256u * p;
        const unsigned t_d1 = t_row + 64u * hw, t_d2 = t_row + 128u + 64u * hw;
        const unsigned* sb1 = reinterpret_cast<const unsigned*>(g + S::B1) + 32 * hw;           // pairs of bf16
        auto piece = [](int jj) { return 32 * jj + (jj >= 2 ? 64 : 0); };                       // its jj-th 32 columns, from 64 hw
        const unsigned* sb2 = reinterpret_cast<const unsigned*>(g + S::B2) + 32 * hw;
        unsigned hk[RES ? 32 : 1];                             // RES: this thread's 64 hidden values, the residual of layer 2
        const unsigned char* xrow = g + S::X + p * X_BYTES + hw * X_SLAB;           // RES: a column half is a slab of the input stage
        unsigned it = 0;
        for (long long tile = first + p * step; tile < a.n_tiles; tile += 2 * step, ++it) {
            const unsigned par = it & 1u;
            if (!__all_sync(0xffffffffu, mbar_wait(bar(D1_FULL + p), par, abort_flag))) { failed = true; break; }   // warp-uniform: the TMEM accesses below are warp-wide
            tc_fence_after();
            // its turn: one tile's activations at a time. Both epilogues want the same unit (MUFU); let run side by side they fall into
            // step and leave it idle while both wait for their contractions
            if ((it > 0 || p == 1) && !__all_sync(0xffffffffu, mbar_wait(bar(TURN + p), p == 1 ? par : par ^ 1u, abort_flag))) { failed = true; break; }
            unsigned raw1[2][32];
            tmem_ld32(t_d1, raw1[0]);
#pragma unroll
            for (int jj = 0; jj < NCH; ++jj) {
                unsigned (&v)[32] = raw1[jj & 1];
                unsigned pk[16];
                tmem_wait_ld();
                if (jj == NCH - 1) mbar_arrive(bar(TURN + (p ^ 1)));                                     // the other tile starts under the last piece
                if (jj + 1 < NCH) tmem_ld32(t_d1 + piece(jj + 1), raw1[(jj + 1) & 1]);                  // on its way under this piece's work
#pragma unroll
                for (int e = 0; e < 16; ++e) {
                    unsigned y = pack2(__uint_as_float(v[2 * e]), __uint_as_float(v[2 * e + 1]));         // matmul -> bf16
                    y = add_bf16x2(y, sb1[piece(jj) / 2 + e]);                                                   // + bias -> bf16 (a null bias is a row of zeros)
                    pk[e] = silu_pair(y);                                                                  // SiLU -> bf16
                }
                if (RES) {                  // + input -> bf16: the thread's own row of the tile, still in its input stage
#pragma unroll
                    for (int e = 0; e < 16; ++e) {
                        pk[e] = add_bf16x2(pk[e], *reinterpret_cast<const unsigned*>(xrow + kmajor_off(row, 32 * jj + 2 * e, TC_TILE)));
                        hk[(16 * jj + e) & (RES ? 31 : 0)] = pk[e];
                    }
                }
                tmem_st16(t_d1 + 16u * jj, pk);               // over columns this warp has read
            }
            tmem_wait_st();
            tc_fence_before();
            mbar_arrive(bar(H_FULL + p));

            if (!__all_sync(0xffffffffu, mbar_wait(bar(D2_FULL + p), par, abort_flag))) { failed = true; break; }
            tc_fence_after();
            unsigned v[2][32];
            tmem_ld32(t_d2, v[0]);
            tmem_ld32(t_d2 + 32u, v[1]);
            tmem_wait_ld();
            tc_fence_before();
            mbar_arrive(bar(D2_FREE + p));
            unsigned word[2];
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                unsigned y[16];
#pragma unroll
                for (int e = 0; e < 16; ++e) {
                    y[e] = add_bf16x2(pack2(__uint_as_float(v[j][2 * e]), __uint_as_float(v[j][2 * e + 1])), sb2[16 * j + e]);
                    if (RES) y[e] = add_bf16x2(y[e], hk[(16 * j + e) & (RES ? 31 : 0)]);   // + the layer's input (the hidden values of the same columns)
                }
                word[j] = signs16(y);
            }
            const long long b = tile / a.tiles_per_b, t = (tile - b * a.tiles_per_b) * TC_TILE + row;
            if (t < a.T) *reinterpret_cast<uint2*>(a.codes + b * a.cs_b + (t * a.H + h) * 4 + 2 * hw) = make_uint2(word[0], word[1]);
        }
    } else if (warp < TC_EPI_WARPS + 2 && lane == 0) {
        // ================= issuing thread of tile in flight p: TMA copies and tensor-core instructions =================
        const int p = warp - TC_EPI_WARPS;
        const unsigned x_s[2] = {base + S::X + p * X_BYTES, base + S::X + p * X_BYTES + X_SLAB}, tm = tmem + 256u * p;
        constexpr unsigned I1 = instr_desc(D1), I2 = instr_desc(128);
        unsigned loads = 0;
        auto coords = [&](long long tile, int& t0, int& b) {
            const long long bb = tile / a.tiles_per_b;
            b = (int)bb;
            t0 = (int)((tile - bb * a.tiles_per_b) * TC_TILE);
        };
        auto load = [&](long long tile) {
            int t0, b;
            coords(tile, t0, b);
            if (LOAD) bulk_wait_read();                       // the stage's rows have left for the cache
            mbar_expect_tx(bar(X_FULL + p), X_BYTES);
            tma_load_4d(x_s[0], &xmap, bar(X_FULL + p), 0, t0, h, b);              // k 0..63 of the 128 rows
            tma_load_4d(x_s[1], &xmap, bar(X_FULL + p), 64, t0, h, b);             // k 64..127
            ++loads;
        };
        long long tile = first + p * step;
        if (tile < a.n_tiles) load(tile);
        unsigned it = 0;
        for (; tile < a.n_tiles; tile += 2 * step, ++it) {
            const unsigned par = it & 1u;
            if (!mbar_wait(bar(X_FULL + p), par, abort_flag)) { failed = true; break; }
            if (it > 0 && !mbar_wait(bar(D2_FREE + p), par ^ 1u, abort_flag)) { failed = true; break; }   // the tile before is out of TMEM
            tc_fence_after();
#pragma unroll
            for (int ks = 0; ks < 8; ++ks) {
                const unsigned bo = (unsigned)(ks >> 2) * ((unsigned)D1 * 128u) + (unsigned)(ks & 3) * 32u;
                mma_ss(tm, smem_desc(x_s[ks >> 2] + (unsigned)(ks & 3) * 32u), smem_desc(base + S::W1 + bo), I1, ks > 0 ? 1u : 0u);
            }
            tc_commit(bar(D1_FULL + p));
            if (LOAD) {
                int t0, b;
                coords(tile, t0, b);
                tma_store_4d(&kdst, x_s[0], 0, t0, h, b);
                tma_store_4d(&kdst, x_s[1], 64, t0, h, b);
                bulk_commit();
            }
            if (!RES) {                                       // layer 1 is over: the stage takes the next rows
                if (!mbar_wait(bar(D1_FULL + p), par, abort_flag)) { failed = true; break; }
                if (tile + 2 * step < a.n_tiles) load(tile + 2 * step);
            }
            if (!mbar_wait(bar(H_FULL + p), par, abort_flag)) { failed = true; break; }
            tc_fence_after();
            if (RES && tile + 2 * step < a.n_tiles) load(tile + 2 * step);         // the input rows have been added
#pragma unroll
            for (int i = 0; i < D1 / 16; ++i) {
                // D1 = 256: the order of the sums stays the one of the kernel before this one (0 1 4 5 8 9 12 13, then 2 3 6 7 ..): codes
                // built by either are the same bit for bit
                const int ks = D1 == 256 ? 4 * ((i & 7) >> 1) + 2 * (i >> 3) + (i & 1) : i;
                const unsigned ho = (unsigned)((ks >> 2) & 1) * 64u + (unsigned)(ks >> 3) * 32u + (unsigned)(ks & 3) * 8u;
                const unsigned bo = (unsigned)(ks >> 2) * (128u * 128u) + (unsigned)(ks & 3) * 32u;
                mma_ts(tm + 128u, tm + ho, smem_desc(base + S::W2 + bo), I2, i > 0 ? 1u : 0u);
            }
            tc_commit(bar(D2_FULL + p));
        }
        if (LOAD) bulk_wait_read();
        if (failed && loads > 0)                              // a copy of ours may still be in flight: let it land (bounded)
            for (unsigned i = 0; i < WAIT_LIMIT && !mbar_test(bar(X_FULL + p), (loads - 1u) & 1u); ++i) __nanosleep(256);
    } else if (LOAD && warp == TC_EPI_WARPS + 2 && lane == 0) {
        failed = !copy_v_rows(base + S::V, bar(V_FULL), vsrc, vdst, a, first, step, h, abort_flag);
    }
    if (failed) {
        *abort_flag = 1;
        if (a.status) *reinterpret_cast<volatile int*>(a.status) = 3;
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == TC_EPI_WARPS) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
}

// ---- the linear hash 128 -> 128 (one contraction per tile): bound by the stream of the input rows, so the kernel
// keeps four input stages in flight and two accumulators in TMEM; two teams of four epilogue warps take alternate
// tiles (a thread reads its row's 128 columns, adds the bias, takes the sign bits and stores the row's 16-byte code).
constexpr int L1_NS = 4;                        // input stages
constexpr int L1_THREADS = (8 + 2) * 32;
constexpr unsigned L1_W = 128 * 128 * 2, L1_OFF_X = L1_W, L1_OFF_V = L1_OFF_X + L1_NS * X_BYTES, L1_OFF_B = L1_OFF_V + VS * V_PIECE,
                   L1_OFF_BAR = L1_OFF_B + 256, L1_OFF_MISC = L1_OFF_BAR + (8 + VS) * 8, L1_SMEM = L1_OFF_MISC + 16 + 1024;

template <bool LOAD>
__global__ void __launch_bounds__(L1_THREADS, 1)
hash_encode_tc_linear_kernel(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap kdst,
                             const __grid_constant__ CUtensorMap vsrc, const __grid_constant__ CUtensorMap vdst, const HashTcArgs a) {
    extern __shared__ unsigned char smem_raw[];
    const unsigned raw = (unsigned)__cvta_generic_to_shared(smem_raw);
    const unsigned base = (raw + 1023u) & ~1023u;
    unsigned char* g = smem_raw + (base - raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int h = blockIdx.y;
    volatile int* abort_flag = reinterpret_cast<volatile int*>(g + L1_OFF_MISC + 4);
    unsigned* tmem_slot = reinterpret_cast<unsigned*>(g + L1_OFF_MISC);
    auto bar = [&](int i) { return base + L1_OFF_BAR + (unsigned)i * 8u; };
    constexpr int X_FULL = 0 /* .. 3 */, D_FULL = 4 /* , 5 */, D_FREE = 6 /* , 7 */, V_FULL = 8 /* .. */;

    if (tid == 0) {
        *abort_flag = 0;
        for (int i = 0; i < L1_NS; ++i) mbar_init(bar(X_FULL + i), 1);
        for (int i = 0; i < VS; ++i) mbar_init(bar(V_FULL + i), 1);
        for (int i = 0; i < 2; ++i) { mbar_init(bar(D_FULL + i), 1); mbar_init(bar(D_FREE + i), 128); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 8) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 256;" ::"r"(base + L1_OFF_MISC) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    {
        const uint4* w1 = reinterpret_cast<const uint4*>(a.w1 + (long long)h * 128 * 128);        // [k][n], 16 groups of 8 n per row
        for (int task = warp; task < 4 * 16; task += L1_THREADS / 32) {
            const int k = (task >> 4) * 32 + lane, n0 = (task & 15) * 8;
            const uint4 v = w1[k * 16 + (task & 15)];
            const unsigned short* e = reinterpret_cast<const unsigned short*>(&v);
#pragma unroll
            for (int c = 0; c < 8; ++c) *reinterpret_cast<unsigned short*>(g + kmajor_off(n0 + c, k, 128)) = e[c];
        }
        __nv_bfloat16* sb = reinterpret_cast<__nv_bfloat16*>(g + L1_OFF_B);
        for (int i = tid; i < 128; i += L1_THREADS) sb[i] = a.b1 ? a.b1[(long long)h * 128 + i] : __float2bfloat16_rn(0.0f);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = *tmem_slot;
    const long long first = blockIdx.x, step = gridDim.x;
    bool failed = false;

    if (warp < 8) {
        // ================= epilogue team `team` takes the CTA's tiles team, team + 2, ... =================
        const int team = warp >> 2, q = warp & 3, row = q * 32 + lane;
        const unsigned t_d = tmem + ((unsigned)(q * 32) << 16) + 128u * team;
        const unsigned* sb = reinterpret_cast<const unsigned*>(g + L1_OFF_B);
        unsigned it = team;
        for (long long tile = first + team * step; tile < a.n_tiles; tile += 2 * step, it += 2) {
            if (!__all_sync(0xffffffffu, mbar_wait(bar(D_FULL + team), (it >> 1) & 1u, abort_flag))) { failed = true; break; }
            tc_fence_after();
            unsigned v[4][32];
#pragma unroll
            for (int j = 0; j < 4; ++j) tmem_ld32(t_d + 32u * j, v[j]);
            tmem_wait_ld();
            tc_fence_before();
            mbar_arrive(bar(D_FREE + team));
            unsigned word[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                unsigned y[16];
#pragma unroll
                for (int e = 0; e < 16; ++e)                                                               // matmul -> bf16, + bias -> bf16
                    y[e] = add_bf16x2(pack2(__uint_as_float(v[j][2 * e]), __uint_as_float(v[j][2 * e + 1])), sb[16 * j + e]);
                word[j] = signs16(y);
            }
            const long long b = tile / a.tiles_per_b, t = (tile - b * a.tiles_per_b) * TC_TILE + row;
            if (t < a.T) *reinterpret_cast<uint4*>(a.codes + b * a.cs_b + (t * a.H + h) * 4) = make_uint4(word[0], word[1], word[2], word[3]);
        }
    } else if (warp == 8 && lane == 0) {
        // ================= issuing thread =================
        const unsigned x_s = base + L1_OFF_X;
        constexpr unsigned I1 = instr_desc(128);
        bool pending[L1_NS] = {false, false, false, false};
        auto load = [&](long long tile, int st) {
            const long long b = tile / a.tiles_per_b;
            const int t0 = (int)((tile - b * a.tiles_per_b) * TC_TILE);
            const unsigned dst = x_s + (unsigned)st * X_BYTES;
            mbar_expect_tx(bar(X_FULL + st), X_BYTES);
            tma_load_4d(dst, &xmap, bar(X_FULL + st), 0, t0, h, (int)b);
            tma_load_4d(dst + X_BYTES / 2, &xmap, bar(X_FULL + st), 64, t0, h, (int)b);
            pending[st] = true;
        };
        for (int i = 0; i < L1_NS; ++i)
            if (first + i * step < a.n_tiles) load(first + i * step, i);
        unsigned it = 0;
        for (long long tile = first; tile < a.n_tiles; tile += step, ++it) {
            const int st = (int)(it % L1_NS), buf = (int)(it & 1u);
            if (!mbar_wait(bar(X_FULL + st), (it / L1_NS) & 1u, abort_flag)) { failed = true; break; }
            pending[st] = false;
            if (it >= 2 && !mbar_wait(bar(D_FREE + buf), ((it >> 1) - 1u) & 1u, abort_flag)) { failed = true; break; }   // the accumulator has been read
            tc_fence_after();
#pragma unroll
            for (int ks = 0; ks < 8; ++ks) {
                const unsigned ao = (unsigned)st * X_BYTES + (unsigned)(ks >> 2) * (X_BYTES / 2) + (unsigned)(ks & 3) * 32u;
                const unsigned bo = (unsigned)(ks >> 2) * (128u * 128u) + (unsigned)(ks & 3) * 32u;
                mma_ss(tmem + 128u * buf, smem_desc(x_s + ao), smem_desc(base + bo), I1, ks > 0 ? 1u : 0u);
            }
            tc_commit(bar(D_FULL + buf));
            if (LOAD) {
                const long long b = tile / a.tiles_per_b;
                const int t0 = (int)((tile - b * a.tiles_per_b) * TC_TILE);
                tma_store_4d(&kdst, x_s + (unsigned)st * X_BYTES, 0, t0, h, (int)b);
                tma_store_4d(&kdst, x_s + (unsigned)st * X_BYTES + X_SLAB, 64, t0, h, (int)b);
                bulk_commit();
            }
            if (it >= 1) {       // the contraction of the tile before this one is over by now or soon: its input stage takes the next rows
                if (!mbar_wait(bar(D_FULL + (buf ^ 1)), ((it - 1u) >> 1) & 1u, abort_flag)) { failed = true; break; }
                const long long nxt = tile + (long long)(L1_NS - 1) * step;
                if (LOAD) bulk_wait_read1();                  // that tile's rows have left for the cache (this one's may still be leaving)
                if (nxt < a.n_tiles) load(nxt, (int)((it - 1u) % L1_NS));
            }
        }
        if (LOAD) bulk_wait_read();
        if (failed) {
            for (int st = 0; st < L1_NS; ++st)
                if (pending[st]) {
                    for (unsigned i = 0; i < WAIT_LIMIT && !(mbar_test(bar(X_FULL + st), 0u) || mbar_test(bar(X_FULL + st), 1u)); ++i) __nanosleep(256);
                }
        }
    } else if (LOAD && warp == 9 && lane == 0) {
        failed = !copy_v_rows(base + L1_OFF_V, bar(V_FULL), vsrc, vdst, a, first, step, h, abort_flag);
    }
    if (failed) {
        *abort_flag = 1;
        if (a.status) *reinterpret_cast<volatile int*>(a.status) = 3;
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 8) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 256;" ::"r"(tmem) : "memory");
}

int* g_status_host = nullptr;     // one mapped host word for the process: any device and any of the tensor-core kernels may raise it
int g_hash_kernel = 0;            // 1: warp-level kernel only; else this kernel whenever it covers the shape

}  // namespace

namespace sl {

void set_hash_kernel(int mode) { g_hash_kernel = mode; }

// The status word as the current device addresses it (null: none to be had). The first call may come from any thread and inside a
// stream capture, which forbids an allocation unless the thread says that it is none of the capture's business.
int* tc_status_word() {
    static std::mutex mu;
    {
        std::lock_guard<std::mutex> lock(mu);
        if (!g_status_host) {
            cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
            cudaThreadExchangeStreamCaptureMode(&mode);
            int* p = nullptr;
            const cudaError_t e = cudaHostAlloc(reinterpret_cast<void**>(&p), sizeof(int), cudaHostAllocMapped | cudaHostAllocPortable);
            cudaThreadExchangeStreamCaptureMode(&mode);
            if (e != cudaSuccess) { cudaGetLastError(); return nullptr; }
            *p = 0;
            g_status_host = p;
        }
    }
    int* d_status = nullptr;
    if (cudaHostGetDevicePointer(reinterpret_cast<void**>(&d_status), g_status_host, 0) != cudaSuccess) { cudaGetLastError(); return nullptr; }
    return d_status;
}

// Returns the hash status word (0, or 3 after a device-side wait ran out) and clears it. The caller synchronises first.
int take_hash_status() {
    if (!g_status_host) return 0;
    const int v = *reinterpret_cast<volatile int*>(g_status_host);
    *reinterpret_cast<volatile int*>(g_status_host) = 0;
    return v;
}

// Returns SL_OK after launching, 1 when the shape is not one this kernel covers (the caller falls through to the
// warp-level kernel), or an error code. With `load` the rows are also stored to the K cache and their V rows copied.
int launch_hash_encode_tc(const void* x, long long xs_b, long long xs_tok, long long xs_h, int B, long long T, int H, const sl_hash_params* hp,
                          uint32_t* codes, long long cs_b, const LoadRows* load, cudaStream_t s) {
    if (g_hash_kernel == 1) return 1;
    const bool mlp = hp->n_layers == 2 && hp->dims[0] == 128 && (hp->dims[1] == 256 || hp->dims[1] == 128) && hp->dims[2] == 128;
    const bool linear = hp->n_layers == 1 && hp->dims[0] == 128 && hp->dims[1] == 128;
    if ((!mlp && !linear) || (hp->residue && (linear || hp->dims[1] != 128))) return 1;
    if (H > 65535 || B > 65535 || T > 0x7fffff00ll) return 1;
    // no lower limit on the rows: from 64 rows up this kernel takes as long as the warp-level one or less (1024 rows of 8 heads: 18.5 us
    // against 32.9 with a hidden layer of 256, 12.7 against 20.9 with 128, equal for the linear hash)
    if (!sl::aligned16(x) || !sl::aligned16(codes) || cs_b % 4 != 0) return 1;
    EncodeTiledFn enc = encode_fn();
    if (!enc) return 1;
    int* d_status = sl::tc_status_word();
    if (!d_status) return 1;

    // a map over [B,T,H,128] rows, boxes of 128 rows x 64 columns in the operands' swizzled layout, or (V) of 32 whole rows as they
    // are; false where TMA cannot address them
    auto encode = [&](CUtensorMap* map, const void* p, long long st_b, long long st_tok, long long st_h, bool operand = true) {
        if (!sl::aligned16(p) || st_tok % 8 != 0 || st_h % 8 != 0 || st_tok < 128 || st_h < 128 || (B > 1 && (st_b % 8 != 0 || st_b <= 0))) return false;
        const cuuint64_t gdim[4] = {128, (cuuint64_t)T, (cuuint64_t)H, (cuuint64_t)B};
        const cuuint64_t gstr[3] = {(cuuint64_t)st_tok * 2, (cuuint64_t)st_h * 2, (cuuint64_t)(B > 1 ? st_b : T * st_tok) * 2};
        const cuuint32_t box[4] = {operand ? 64u : 128u, operand ? (unsigned)TC_TILE : 32u, 1, 1}, estr[4] = {1, 1, 1, 1};
        return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(p), gdim, gstr, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   operand ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
    };
    CUtensorMap map, kdst, vsrc, vdst;
    if (!encode(&map, x, xs_b, xs_tok, xs_h)) return 1;
    kdst = vsrc = vdst = map;
    if (load && (!encode(&kdst, load->k_cache, load->cs_b, load->cs_tok, load->cs_h) ||
                 !encode(&vsrc, load->v, load->vs_b, load->vs_tok, load->vs_h, false) ||
                 !encode(&vdst, load->v_cache, load->cs_b, load->cs_tok, load->cs_h, false)))
        return 1;

    HashTcArgs a = {};
    a.T = T; a.H = H; a.B = B;
    a.w1 = static_cast<const __nv_bfloat16*>(hp->d_w[0]); a.b1 = static_cast<const __nv_bfloat16*>(hp->d_b[0]);
    if (mlp) { a.w2 = static_cast<const __nv_bfloat16*>(hp->d_w[1]); a.b2 = static_cast<const __nv_bfloat16*>(hp->d_b[1]); }
    a.codes = codes; a.cs_b = cs_b;
    a.tiles_per_b = (T + TC_TILE - 1) / TC_TILE;
    a.n_tiles = a.tiles_per_b * B;
    a.status = d_status;
    const long long per_head = std::max<long long>(1, (long long)sl::sm_count() / H);
    const unsigned gx = (unsigned)std::min<long long>(a.n_tiles, per_head);
    typedef void (*Kern)(const CUtensorMap, const CUtensorMap, const CUtensorMap, const CUtensorMap, const HashTcArgs);
    Kern kern;
    unsigned smem, threads = TC_THREADS;
    if (!mlp) {
        kern = load ? (Kern)hash_encode_tc_linear_kernel<true> : (Kern)hash_encode_tc_linear_kernel<false>;
        smem = L1_SMEM; threads = L1_THREADS;
    } else if (hp->dims[1] == 256) {
        kern = load ? (Kern)hash_encode_tc_kernel<256, false, true> : (Kern)hash_encode_tc_kernel<256, false, false>;
        smem = TcSmem<256>::BYTES;
    } else {
        if (hp->residue) kern = load ? (Kern)hash_encode_tc_kernel<128, true, true> : (Kern)hash_encode_tc_kernel<128, true, false>;
        else kern = load ? (Kern)hash_encode_tc_kernel<128, false, true> : (Kern)hash_encode_tc_kernel<128, false, false>;
        smem = TcSmem<128>::BYTES;
    }
    SL_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kern<<<dim3(gx, (unsigned)H), threads, smem, s>>>(map, kdst, vsrc, vdst, a);
    SL_CUDA_OK(cudaGetLastError());
    return SL_OK;
}

}  // namespace sl

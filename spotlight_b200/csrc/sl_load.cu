// New rows into a layer's caches (sl_load_rows). Without their codes, or where the tensor-core kernel does not build them: K and V in one
// launch, 16-byte pieces, four in flight per thread. Bound by its bytes: 131 072 x 8 rows of K and V (1.07 GB moved) in 177 us, 6.1 TB/s
// (two strided torch copies: 594 us).
// A module of its own (see sl_attn_dense.cu). Few rows without codes stay with two copies of the caller's (session.py).
#include "sl_common.cuh"

namespace {
struct CopyRowsArgs {
    const unsigned char* src[2]; unsigned char* dst[2];
    long long ss_b[2], ss_tok[2], ss_h[2], ds_b, ds_tok, ds_h;      // bytes
    unsigned T, KH; int lg;                                          // 1 << lg 16-byte pieces per row
};

__global__ void __launch_bounds__(256) copy_rows_kernel(const CopyRowsArgs a) {
    const int w = blockIdx.z, b = blockIdx.y;
    const long long ss_tok = w ? a.ss_tok[1] : a.ss_tok[0], ss_h = w ? a.ss_h[1] : a.ss_h[0];
    const unsigned char* src = (w ? a.src[1] : a.src[0]) + (long long)b * (w ? a.ss_b[1] : a.ss_b[0]);
    unsigned char* dst = (w ? a.dst[1] : a.dst[0]) + (long long)b * a.ds_b;
    const long long n = ((long long)a.T * a.KH) << a.lg, stride = (long long)gridDim.x * 256;
    for (long long i0 = (long long)blockIdx.x * 256 + threadIdx.x; i0 < n; i0 += 4 * stride) {
        uint4 v[4];
        long long to[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const long long i = i0 + u * stride;
            if (i < n) {
                const long long r = i >> a.lg, t = r / a.KH, h = r - t * a.KH, c = (i & ((1 << a.lg) - 1)) << 4;
                v[u] = sl::ld_stream_v4(reinterpret_cast<const uint4*>(src + t * ss_tok + h * ss_h + c));
                to[u] = t * a.ds_tok + h * a.ds_h + c;
            }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (i0 + u * stride < n) *reinterpret_cast<uint4*>(dst + to[u]) = v[u];
    }
}
}  // namespace

extern "C" int sl_load_rows(const void* d_k, const sl_kv_layout* k_src, const void* d_v, const sl_kv_layout* v_src, int dtype, int B, int64_t T,
                            int KH, void* d_k_cache, void* d_v_cache, const sl_kv_layout* kv, const sl_hash_params* hash,
                            uint32_t* d_codes, int64_t code_batch_stride, void* stream) {
    SL_REQUIRE(d_k && d_v && k_src && v_src && d_k_cache && d_v_cache && kv && (!hash || d_codes), SL_EINVAL, "sl_load_rows: null pointer");
    SL_REQUIRE(B > 0 && B <= 65535 && T >= 0 && T <= 0x7fffff00ll && KH > 0, SL_ESHAPE, "sl_load_rows: bad shape");
    SL_REQUIRE(dtype == SL_BF16 || dtype == SL_F16 || dtype == SL_F32, SL_EINVAL, "sl_load_rows: unknown dtype %d", dtype);
    const int es = dtype == SL_F32 ? 4 : 2;
    const void* ptrs[4] = {d_k, d_v, d_k_cache, d_v_cache};
    const sl_kv_layout* lay[4] = {k_src, v_src, kv, kv};
    for (int i = 0; i < 4; ++i) {
        SL_REQUIRE(sl::aligned16(ptrs[i]) && lay[i]->batch_stride * es % 16 == 0 && lay[i]->token_stride * es % 16 == 0 &&
                   lay[i]->head_stride * es % 16 == 0, SL_EALIGN, "sl_load_rows: rows not 16-byte aligned");
        SL_REQUIRE(lay[i]->batch_stride >= 0 && lay[i]->token_stride >= 0 && lay[i]->head_stride >= 0 &&
                   (i < 2 || (lay[i]->token_stride >= 128 && lay[i]->head_stride >= 128)), SL_ESHAPE, "sl_load_rows: strides");
    }
    if (hash) {
        if (int rc = sl::check_hash_params("sl_load_rows", hash, dtype)) return rc;
        SL_REQUIRE(code_batch_stride >= T * KH * 4, SL_ESHAPE, "sl_load_rows: code batch stride shorter than a batch row");
    }
    if (T == 0) return SL_OK;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (hash && dtype == SL_BF16 && (long long)B * T >= 64) {
        const sl::LoadRows load = {d_k_cache, d_v_cache, kv->batch_stride, kv->token_stride, kv->head_stride,
                                   d_v, v_src->batch_stride, v_src->token_stride, v_src->head_stride};
        const int rt = sl::launch_hash_encode_tc(d_k, k_src->batch_stride, k_src->token_stride, k_src->head_stride, B, T, KH, hash, d_codes,
                                                 code_batch_stride, &load, s);
        if (rt <= 0) return rt;
    }
    CopyRowsArgs a = {};
    for (int i = 0; i < 2; ++i) {
        a.src[i] = static_cast<const unsigned char*>(ptrs[i]);
        a.dst[i] = static_cast<unsigned char*>(const_cast<void*>(ptrs[2 + i]));
        a.ss_b[i] = lay[i]->batch_stride * es; a.ss_tok[i] = lay[i]->token_stride * es; a.ss_h[i] = lay[i]->head_stride * es;
    }
    a.ds_b = kv->batch_stride * es; a.ds_tok = kv->token_stride * es; a.ds_h = kv->head_stride * es;
    a.T = (unsigned)T; a.KH = (unsigned)KH; a.lg = es == 4 ? 5 : 4;
    const long long want = ((T * KH << a.lg) + 1023) / 1024, cap = std::max<long long>(1, (long long)sl::sm_count() * 8 / (2 * B));
    copy_rows_kernel<<<dim3((unsigned)std::min(want, cap), (unsigned)B, 2), 256, 0, s>>>(a);
    SL_CUDA_OK(cudaGetLastError());
    if (!hash) return SL_OK;
    return sl_hash_encode_ex(d_k_cache, kv->batch_stride, kv->token_stride, kv->head_stride, dtype, B, T, KH, hash, d_codes, code_batch_stride, stream);
}

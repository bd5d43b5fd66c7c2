// The merge of the attention kernels' per-split partials (sl_attn_mma.cuh, sl_attn.cu), a module of its own: every long decode
// step runs it, and beside the many forms of the scalar kernel its place moved with each of them (the 32-layer step at 128K keys
// ran 0.7 % behind its former time there, 0.3 % here).
#include "sl_attn.cuh"

namespace {

// One CTA per query head merges the partials of its splits: thread (grp, col) accumulates the
// splits s = grp (mod 4) of output column col with every load in flight at once.
template <typename T>
__global__ void __launch_bounds__(512) attn_merge_kernel(const float* __restrict__ part, int splits, int G, int KH,
                                                         int layout, T* __restrict__ out, float* __restrict__ lse) {
    __shared__ float s_m[sl::ATTN_MAX_SPLITS], s_l[sl::ATTN_MAX_SPLITS], s_w[sl::ATTN_MAX_SPLITS];
    __shared__ float red[4][128];
    sl::pdl_trigger();
    sl::pdl_wait();
    const int g = blockIdx.x % G;
    const long long bh = blockIdx.x / G;
    const int h = (int)(bh % KH);
    const long long b = bh / KH;
    const int tid = threadIdx.x, col = tid & 127, grp = tid >> 7;
    const float* pb = part + (bh * splits * G + g) * 130;             // split s at pb + s*G*130
    const long long sstride = (long long)G * 130;
    float v[sl::ATTN_MAX_SPLITS / 4];
#pragma unroll
    for (int j = 0; j < sl::ATTN_MAX_SPLITS / 4; ++j) {
        const int s = grp + 4 * j;
        v[j] = s < splits ? __ldcg(pb + s * sstride + col) : 0.0f;
    }
    if (tid < splits) {
        s_m[tid] = __ldcg(pb + tid * sstride + 128);
        s_l[tid] = __ldcg(pb + tid * sstride + 129);
    }
    __syncthreads();
    float M = -INFINITY;
    for (int s = 0; s < splits; ++s) M = fmaxf(M, s_m[s]);
    if (tid < splits) s_w[tid] = M == -INFINITY ? 0.0f : exp2f(s_m[tid] - M);
    __syncthreads();
    float acc = 0.0f;
#pragma unroll
    for (int j = 0; j < sl::ATTN_MAX_SPLITS / 4; ++j) {
        const int s = grp + 4 * j;
        if (s < splits) acc = fmaf(v[j], s_w[s], acc);
    }
    red[grp][col] = acc;
    __syncthreads();
    if (grp == 0) {
        float L = 0.0f;
        for (int s = 0; s < splits; ++s) L = fmaf(s_l[s], s_w[s], L);
        const float O = (red[0][col] + red[1][col]) + (red[2][col] + red[3][col]);
        const int qh = layout == SL_GQA_INTERLEAVED ? g * KH + h : h * G + g;
        const long long o = ((long long)b * KH * G + qh) * 128 + col;
        out[o] = sl::VT<T>::from_f(L > 0.0f ? O / L : 0.0f);
        if (lse && col == 0) lse[(long long)b * KH * G + qh] = L > 0.0f ? (M + log2f(L)) * LN2 : -INFINITY;
    }
}

}  // namespace

namespace sl {
int launch_attn_merge(const AttnArgs& a, int G, int dtype, cudaStream_t s) {
    const unsigned blocks = (unsigned)(a.B * a.KH * G);
    switch (dtype) {
        case SL_BF16: SL_CUDA_OK(launch_kernel(attn_merge_kernel<__nv_bfloat16>, dim3(blocks), dim3(512), 0, s, false, (const float*)a.part, a.splits, G, a.KH, a.layout, (__nv_bfloat16*)a.out, a.lse)); break;
        case SL_F16: SL_CUDA_OK(launch_kernel(attn_merge_kernel<__half>, dim3(blocks), dim3(512), 0, s, false, (const float*)a.part, a.splits, G, a.KH, a.layout, (__half*)a.out, a.lse)); break;
        default: SL_CUDA_OK(launch_kernel(attn_merge_kernel<float>, dim3(blocks), dim3(512), 0, s, false, (const float*)a.part, a.splits, G, a.KH, a.layout, (float*)a.out, a.lse)); break;
    }
    return SL_OK;
}
}  // namespace sl

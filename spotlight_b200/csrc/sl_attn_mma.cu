// The tensor-core decode attention (sl_attn_mma.cuh) over index lists and in fill mode, and the rules of its launches.
#include "sl_attn_mma.cuh"

namespace sl {

static int g_attn_warps = 0;        // 0: by shape; 4 / 8: forced (sl_configure, for measurements)
static int g_attn_cluster = 1;      // 1: combine the splits inside a thread-block cluster where one fits; 0: always the merge kernel
void set_attn_warps(int v) { g_attn_warps = v; }
void set_attn_cluster(int v) { g_attn_cluster = v; }
bool fat_ctas(int B, int KH) { return g_attn_warps ? g_attn_warps == 8 : B * KH <= sm_count(); }

// How many clusters of cs CTAs of MW warps the device holds at once (0: none, or the query failed); cached.
template <int MW>
static int max_clusters(int cs) {
    static int cache[17] = {};                         // 0 = not asked yet, -1 = none
    if (cs < 2 || cs > 16) return 0;
    if (cache[cs] == 0) {
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute attrs[2];
        int n = 0;
        if (cluster_config<false, MW, false, false>(cfg, attrs, cs, 1, 1, nullptr) != cudaSuccess ||
            cudaOccupancyMaxActiveClusters(&n, reinterpret_cast<const void*>(sparse_attn_mma_kernel<false, MW, true, false, false>), &cfg) != cudaSuccess) {
            cudaGetLastError();
            n = 0;
        }
        cache[cs] = n > 0 ? n : -1;
    }
    return cache[cs] > 0 ? cache[cs] : 0;
}

// The splits of a (row, head) pair form one cluster when all the clusters of the launch fit on the device at once.
bool use_cluster(int B, int KH, int splits) {
    if (!g_attn_cluster || splits < 2 || splits > 16) return false;
    const int have = fat_ctas(B, KH) ? max_clusters<8>(splits) : max_clusters<4>(splits);
    return have >= B * KH;
}

int attn_mma_splits(int B, int KH, int cap, int reserve_sms) {
    // never more CTAs than fit at once (one of eight warps per SM, or two of four); every warp
    // should get at least one 16-row tile
    const int ctas = B * KH;
    const int tiles = (cap + 15) / 16;
    const int mw = fat_ctas(B, KH) ? 8 : 4;
    int s = ((8 / mw) * std::max(1, sm_count() - reserve_sms)) / ctas;    // reserve_sms: left to a kernel that runs beside this one
    s = std::min(s, std::min(ATTN_MAX_SPLITS, std::max(1, tiles / mw)));
    s = std::max(s, 1);
    // a few more keys per CTA are cheaper than partials in global memory and a merge kernel
    if (s > 16 && s <= 24 && use_cluster(B, KH, 16)) s = 16;
    else if (s > 8 && tiles <= 12 * s) {
        // short lists (at most a tile or two per warp) are bound by latency, not by bandwidth: fewer, fatter CTAs in the
        // largest cluster whose copies all fit at once save the merge kernel (measured at 98 % pruning of 128K keys:
        // 10.2 -> 8.0 us; at 90 % the same move costs bandwidth: 34.0 -> 35.1 us for the step)
        for (int cs = std::min(s, 16); cs >= 8; --cs)
            if (use_cluster(B, KH, cs)) { s = cs; break; }
    }
    return s;
}

int attn_cluster_capacity(int warps, int cs) { return warps == 8 ? max_clusters<8>(cs) : max_clusters<4>(cs); }

int launch_attn_mma(const AttnArgs& a, int G, cudaStream_t s) {
    if (!a.idx) return launch_attn_dense(a, G, s);
    return a.tok ? launch_by_shape<true, false>(a, G, s) : launch_by_shape<false, false>(a, G, s);
}

}  // namespace sl

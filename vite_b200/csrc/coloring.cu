// distColoringMultiHashMinMax for one rank (coloring.cpp:52-118). Each round of
// distColoringIteration (coloring.cpp:133-247) only compares hashes against
// neighbours that are uncolored or colored in this round, so a round is
// order-independent; here one thread colors one vertex and a round is one launch.
#include "vg_internal.cuh"

namespace {

constexpr int MAX_HASH = 32;
constexpr int64_t COLOR_HASH_NE = 1 << 17;

// coloring.cpp:120-131
__host__ __device__ __forceinline__ uint32_t color_hash(uint32_t a, uint32_t seed) {
    a ^= seed;
    a = (a + 0x7ed55d16u) + (a << 12);
    a = (a ^ 0xc761c23cu) + (a >> 19);
    a = (a + 0x165667b1u) + (a << 5);
    a = (a ^ 0xd3a2646cu) + (a << 9);
    a = (a + 0xfd7046c5u) + (a << 3);
    a = (a ^ 0xb55a4f09u) + (a >> 16);
    return a;
}

// one round; colors of this round are >= nextColor, so reading a neighbour
// colored concurrently in this round gives the same decision as reading -1
__global__ void k_color_round(const int64_t *__restrict__ rowptr, const int32_t *__restrict__ tail,
                              int64_t nv, int32_t *__restrict__ color, int nHash, int64_t nextColor,
                              uint32_t seed, unsigned long long *__restrict__ ncolored,
                              const int32_t *__restrict__ ref) {
    unsigned long long mine = 0;
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < nv;
         v += (int64_t)gridDim.x * blockDim.x) {
        if (color[v] != -1) continue;
        // hashes and the color pick use reference ids (v + base of the reference)
        const int64_t rv = vg_rid(ref, (int32_t)v);
        int64_t possible = 2 * (int64_t)nHash;
        uint32_t vHash[MAX_HASH];
        for (int t = 0; t < nHash; t++)
            vHash[t] = color_hash((uint32_t)rv, (uint32_t)((int64_t)seed + 1043 * (int64_t)t));
        uint32_t not_min = 0, not_max = 0;
        bool can_color = true;
        const int64_t e1 = rowptr[v + 1];
        for (int64_t k = rowptr[v]; k < e1; k++) {
            const int32_t u = tail[k];
            if (u == v) continue;
            const int32_t cu = color[u];
            if (cu != -1 && cu < nextColor) continue;
            for (int t = 0; t < nHash; t++) {
                const uint32_t j = color_hash((uint32_t)vg_rid(ref, u),
                                              (uint32_t)((int64_t)seed + 1043 * (int64_t)t));
                if (vHash[t] <= j && !(not_max & (1u << t))) {
                    not_max |= (1u << t);
                    possible--;
                }
                if (vHash[t] >= j && !(not_min & (1u << t))) {
                    not_min |= (1u << t);
                    possible--;
                }
            }
            if (possible == 0) {
                can_color = false;
                break;
            }
        }
        if (can_color) {
            const int64_t col_id = rv % possible;
            int64_t this_col = 0;
            for (int t = 0; t < nHash; t++) {
                if (!(not_min & (1u << t)) && col_id == this_col) {
                    color[v] = (int32_t)(2 * t + nextColor);
                    mine++;
                    break;
                }
                this_col += !(not_min & (1u << t));
                if (!(not_max & (1u << t)) && col_id == this_col) {
                    color[v] = (int32_t)(2 * t + 1 + nextColor);
                    mine++;
                    break;
                }
                this_col += !(not_max & (1u << t));
            }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mine += __shfl_down_sync(0xffffffffu, mine, o);
    if ((threadIdx.x & 31) == 0 && mine) atomicAdd(ncolored, mine);
}

// The round's hashes of every vertex, P (4 or 8) words each, so that a round reads a
// neighbour's in one 16- or 32-byte load instead of computing them once per entry (the
// hashes were two thirds of a round's instructions).
template <int P>
__global__ void k_color_hash(int64_t nv, int nHash, uint32_t seed, const int32_t *__restrict__ ref,
                             uint32_t *__restrict__ hash) {
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < nv;
         v += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t r = (uint32_t)vg_rid(ref, (int32_t)v);
        uint4 h[P / 4];
#pragma unroll
        for (int q = 0; q < P / 4; q++) {
            auto one = [&](int t) { // hashes past nHash are never looked at
                return t < nHash ? color_hash(r, (uint32_t)((int64_t)seed + 1043 * (int64_t)t)) : 0u;
            };
            h[q] = make_uint4(one(4 * q), one(4 * q + 1), one(4 * q + 2), one(4 * q + 3));
        }
#pragma unroll
        for (int q = 0; q < P / 4; q++) reinterpret_cast<uint4 *>(hash)[v * (P / 4) + q] = h[q];
    }
}

// k_color_round with the hashes read from k_color_hash's array. A warp takes 32 vertices, whose
// rows are one range of entries, and reads the tails of a range of up to CR_STAGE entries
// together into shared memory (a lane per row touches a line per lane and load). A vertex
// stops once every hash has a smaller and a larger neighbour. FIRST: no vertex has a color of
// an earlier round, so the neighbours' colors are not read.
constexpr int CR_WARPS = 8, CR_STAGE = 768;
template <int P, bool FIRST>
__global__ void __launch_bounds__(CR_WARPS * 32) k_color_round_hashed(
    const int64_t *__restrict__ rowptr, const int32_t *__restrict__ tail, int64_t nv,
    int32_t *color, int nHash, int64_t nextColor, const uint32_t *__restrict__ hash,
    unsigned long long *__restrict__ ncolored, const int32_t *__restrict__ ref) {
    __shared__ int32_t s_tail[CR_WARPS][CR_STAGE];
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    int32_t *st = s_tail[threadIdx.x >> 5];
    const uint4 *__restrict__ h4 = reinterpret_cast<const uint4 *>(hash);
    const uint32_t all = (1u << nHash) - 1u;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    unsigned mine = 0;
    for (int64_t tile = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; tile * 32 < nv; tile += nw) {
        const int64_t v = tile * 32 + lane;
        const bool valid = v < nv;
        const bool open = valid && (FIRST || color[v] == -1);
        if (!__any_sync(full, open)) continue;
        int64_t e0 = 0, e1 = 0;
        if (valid) {
            e0 = rowptr[v];
            e1 = rowptr[v + 1];
        }
        const int64_t E0 = __shfl_sync(full, e0, 0);
        const int64_t E1 = __shfl_sync(full, e1, 31 - __clz(__ballot_sync(full, valid)));
        const bool staged = E1 - E0 <= CR_STAGE;
        if (staged) {
            for (int j = lane; j < (int)(E1 - E0); j += 32) st[j] = tail[E0 + j];
            __syncwarp();
        }
        if (open) {
            uint32_t own[P];
#pragma unroll
            for (int q = 0; q < P / 4; q++) {
                const uint4 x = h4[v * (P / 4) + q];
                own[4 * q] = x.x;
                own[4 * q + 1] = x.y;
                own[4 * q + 2] = x.z;
                own[4 * q + 3] = x.w;
            }
            uint32_t not_min = 0, not_max = 0;
            bool can_color = true;
            for (int64_t k = e0; k < e1; k++) {
                const int32_t u = staged ? st[k - E0] : tail[k];
                if (u == v) continue;
                if (!FIRST) {
                    const int32_t cu = color[u];
                    if (cu != -1 && cu < nextColor) continue;
                }
#pragma unroll
                for (int q = 0; q < P / 4; q++) {
                    const uint4 x = h4[(int64_t)u * (P / 4) + q];
                    const uint32_t h[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
                    for (int t = 0; t < 4; t++) {
                        not_max |= (uint32_t)(own[4 * q + t] <= h[t]) << (4 * q + t);
                        not_min |= (uint32_t)(own[4 * q + t] >= h[t]) << (4 * q + t);
                    }
                }
                if ((not_max & not_min & all) == all) {
                    can_color = false;
                    break;
                }
            }
            if (can_color) {
                const int64_t rv = vg_rid(ref, (int32_t)v);
                const int possible = __popc(~not_min & all) + __popc(~not_max & all);
                const int64_t col_id = rv % possible;
                int64_t this_col = 0;
                for (int t = 0; t < nHash; t++) {
                    if (!(not_min & (1u << t)) && col_id == this_col) {
                        color[v] = (int32_t)(2 * t + nextColor);
                        mine++;
                        break;
                    }
                    this_col += !(not_min & (1u << t));
                    if (!(not_max & (1u << t)) && col_id == this_col) {
                        color[v] = (int32_t)(2 * t + 1 + nextColor);
                        mine++;
                        break;
                    }
                    this_col += !(not_max & (1u << t));
                }
            }
        }
        __syncwarp();
    }
    mine = __reduce_add_sync(full, mine);
    if (lane == 0 && mine) atomicAdd(ncolored, (unsigned long long)mine);
}

template <int P>
void color_round_hashed(vg_ctx *ctx, const vg_graph *g, int nHash, int64_t nextColor, uint32_t seed,
                        uint32_t *hash, unsigned long long *ncolored) {
    const int64_t nv = g->nv;
    {
        LaunchTimer lt(ctx);
        k_color_hash<P><<<vg_grid(ctx, nv, 256), 256, 0, ctx->stream>>>(nv, nHash, seed, g->ref, hash);
    }
    VG_CHECK_LAUNCH();
    LaunchTimer lt(ctx);
    auto *round = nextColor == 0 ? k_color_round_hashed<P, true> : k_color_round_hashed<P, false>;
    round<<<vg_grid(ctx, nv, CR_WARPS * 32), CR_WARPS * 32, 0, ctx->stream>>>(
        g->rowptr, g->tail, nv, g->colors, nHash, nextColor, hash, ncolored, g->ref);
}

__global__ void k_fill_i32(int32_t *__restrict__ x, int64_t n, int32_t val) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        x[i] = val;
}

} // namespace

void vg_download_comm(vg_ctx *ctx, const int32_t *comm, int64_t n, int64_t *out);
void vg_upload_ids(vg_ctx *ctx, const int64_t *in, int64_t n, int64_t lim, int32_t *out);

// returns nextColor; the colors land in g->colors
int64_t vg_color_internal(vg_ctx *ctx, vg_graph *g, int64_t nHash, int32_t target_percent,
                          int32_t single_iteration) {
    VG_REQUIRE(nHash >= 1 && nHash <= MAX_HASH, "number of hash functions must be 1..%d (got %lld)",
               MAX_HASH, (long long)nHash);
    const int64_t nv = g->nv;
    if (!g->colors) g->colors = (int32_t *)vg_alloc(ctx, sizeof(int32_t) * (nv ? nv : 1));
    if (nv) {
        LaunchTimer lt(ctx);
        k_fill_i32<<<vg_grid(ctx, nv, 256), 256, 0, ctx->stream>>>(g->colors, nv, -1);
    }
    VG_CHECK_LAUNCH();
    DevBuf<unsigned long long> cnt(ctx, 1);
    unsigned long long *h = (unsigned long long *)vg_pinned(ctx, sizeof(unsigned long long));
    // Up to eight hashes are kept per vertex, where there is room for them; below COLOR_HASH_NE
    // entries their launch costs more than it saves (a coloring of some 3,000 vertices
    // 205 -> 219 us).
    DevBuf<uint32_t> hash;
    if (nHash <= 8 && g->ne >= COLOR_HASH_NE) hash.try_alloc(ctx, (size_t)nv * (nHash <= 4 ? 4 : 8));
    uint32_t seed = 1012; // coloring.cpp:60
    int64_t nextColor = 0, lastCount = 0, currentCount = 0;
    const int64_t targetCount = (nv * target_percent) / 100;
    bool finished = false;
    while (!finished) {
        VG_CUDA(cudaMemsetAsync(cnt.p, 0, sizeof(unsigned long long), ctx->stream));
        if (nv && hash.p && nHash <= 4) {
            color_round_hashed<4>(ctx, g, (int)nHash, nextColor, seed, hash.p, cnt.p);
        } else if (nv && hash.p) {
            color_round_hashed<8>(ctx, g, (int)nHash, nextColor, seed, hash.p, cnt.p);
        } else if (nv) {
            LaunchTimer lt(ctx);
            k_color_round<<<vg_grid(ctx, nv, 256), 256, 0, ctx->stream>>>(
                g->rowptr, g->tail, nv, g->colors, (int)nHash, nextColor, seed, cnt.p, g->ref);
        }
        VG_CHECK_LAUNCH();
        VG_CUDA(cudaMemcpyAsync(h, cnt.p, sizeof(*h), cudaMemcpyDeviceToHost, ctx->stream));
        vg_sync(ctx);
        currentCount += (int64_t)*h; // countUnassigned (coloring.cpp:468-491)
        finished = single_iteration || currentCount >= targetCount || lastCount == currentCount;
        nextColor += nHash * 2;
        seed = color_hash(seed, 0);
        lastCount = currentCount;
    }
    g->num_colors = nextColor;
    return nextColor;
}

extern "C" vg_status vg_color(vg_ctx *ctx, vg_graph *g, int64_t n_hash, int32_t target_percent,
                              int32_t single_iteration, int64_t *colors_out,
                              int64_t *num_colors_out) {
    if (!ctx || !g) return VG_ERR_ARG;
    return vg_guard(ctx, [&] {
        VG_CUDA(cudaSetDevice(ctx->device));
        const int64_t nc = vg_color_internal(ctx, g, n_hash, target_percent, single_iteration);
        if (num_colors_out) *num_colors_out = nc;
        if (colors_out) vg_download_vals_ref(ctx, g, g->colors, colors_out);
    });
}

extern "C" vg_status vg_set_colors(vg_ctx *ctx, vg_graph *g, const int64_t *colors,
                                   int64_t num_colors) {
    if (!ctx || !g || !colors) return VG_ERR_ARG;
    return vg_guard(ctx, [&] {
        VG_CUDA(cudaSetDevice(ctx->device));
        VG_REQUIRE(num_colors >= 0 && num_colors < INT32_MAX, "bad number of colors");
        if (!g->colors) g->colors = (int32_t *)vg_alloc(ctx, sizeof(int32_t) * (g->nv ? g->nv : 1));
        vg_upload_ids(ctx, colors, g->nv, num_colors + 1, g->colors);
        vg_ref_to_pos_inplace(ctx, g, g->colors, false);
        g->num_colors = num_colors;
    });
}

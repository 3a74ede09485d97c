// The next level's graph of a small graph in one launch and a copy (included by
// aggregate.cu).
//
// What bounds a small rebuild is its steps: renumbering, grouping, the segments' tables,
// scans and compaction are some 30 launches with three read-backs, 150-590 us for levels
// whose entries take a few microseconds to read. Here the steps run between the barriers
// of one launch (grid_sync.cuh); the host waits once for the new sizes and a second kernel
// copies the rows into arrays of exactly those sizes. Members are put in reference order
// inside their row by sorting each row's own list (in registers up to 32, else through a
// bitmap of the vertices), which replaces the radix sort of all vertices.
//
// Measured, by launches -> here (vertices / entries): 1,201 / 8,082 185 -> 61 us; 2,324 /
// 244,610 585 -> 183 us; 31,145 / 250,126 361 -> 114 us; 90,768 / 617,959 417 -> 143 us. A
// long segment's entries dealt out to the warps: with every warp reading all of them the
// second took 547 us. The line at 2^21 entries keeps the scratch small (24 bytes an entry).
//
// Results as vg_aggregate_rows: rows and keys by first appearance in reference order, every
// sum a left fold in (vertex, entry) order, bit for bit.

#ifndef VG_RS_MAX_NV
#define VG_RS_MAX_NV 131072
#endif
#ifndef VG_RS_MAX_NE
#define VG_RS_MAX_NE (1 << 21)
#endif
#ifndef VG_RS_CLUSTER_NE
#define VG_RS_CLUSTER_NE 16384
#endif
#ifndef VG_RS_NE_PER_CTA
#define VG_RS_NE_PER_CTA 1024
#endif
constexpr int64_t RS_MAX_NV = VG_RS_MAX_NV;
constexpr int64_t RS_MAX_NE = VG_RS_MAX_NE;
static_assert(RS_MAX_NV <= NARROW_KEYS, "warp_segment is told so");
constexpr int RS_BIG_L = 1024; // segments longer than this go to a whole block
// One block reads a long segment while the others wait at the barrier, and one of many keys
// once per 4,096 key values. A graph with a segment that might be read for more entries than this
// is left to the general path before any is read. Whole rebuilds here and by launches: integral
// weights and one read, where the warps share every key, 180,000 entries 0.82 and 0.73 ms, 400,000
// 1.08 and 0.96; several reads, 49,000 entries in all 0.50 and 0.53, 71,000 0.56 and 0.50, 124,000
// 0.70 and 0.47; real weights and one read, where a key's entries are one warp's chain, 24,000
// entries 0.36 and 0.54, 48,000 0.65 and 0.55, 96,000 1.8 and 0.8, 800,000 14.3 and 3.1.
__host__ __device__ __forceinline__ int64_t rs_max_reads(bool integral, int64_t reads) {
    return reads > 1 ? 49152 : integral ? 131072 : 32768;
}

using SmallWarpTable = HashWarpSmem<H_CAP, H_MAXU>;
using SmallBlockTable = BlockTableLarge;
static_assert(SmallBlockTable::THREADS == GS_THREADS, "the block table's warps are the block's");
constexpr size_t RS_SMEM_BYTES = sizeof(SmallBlockTable) > GS_WARPS * sizeof(SmallWarpTable)
                                     ? sizeof(SmallBlockTable)
                                     : GS_WARPS * sizeof(SmallWarpTable);
static_assert(RS_SMEM_BYTES >= RS_MAX_NV / 8, "the member bitmap must fit");

struct SmallRebuildOut {
    int64_t nc, m; // rows and entries of the next level
    int32_t status;
    int32_t longest; // entries of its longest row
};

struct SmallRebuild {
    int64_t nv, ne;
    int32_t integral; // the weights' sums are exact in any order
    const int64_t *rowptr;
    const int32_t *tail;
    const double *weight;
    const int32_t *ref, *pos; // null: positions are the reference ids
    const int32_t *comm;
    int32_t *first_ref, *first_pos; // per community: first members, then new id and position
    int32_t *next_ref, *next_pos;   // (with a layout) the next level's maps
    int32_t *mcount, *mfill, *mlist; // members per row; their reference ids, row by row
    int64_t *mbase, *rstart, *ecount, *moff, *ucount, *rowptr_out; // nv + 1 each
    int32_t *biglist;  // rows with more than 32 members
    int32_t *longlist; // segments a block takes
    int32_t *ctl;      // RS_CTL words
    int64_t *part;     // 3 per block
    int32_t *gk, *uk;
    double *gw, *uw;
    unsigned *arrived; // as in SmallPhase
    int32_t polls;
    SmallRebuildOut *out;
};
enum { RS_BIG_ROWS, RS_LONG_SEGS, RS_REFUSED, RS_LONGEST, RS_CTL };

// sum of part[0..n) with stride 3, n <= the block's threads; the whole block calls it
__device__ __forceinline__ int64_t block_prefix_of(const int64_t *part, int n, int64_t *s_w) {
    int64_t total;
    block_excl((int)threadIdx.x < n ? __ldcg(part + 3 * threadIdx.x) : 0, total, s_w);
    return total;
}

template <bool GRID>
__global__ void __launch_bounds__(GS_THREADS, 1) k_rebuild_small(SmallRebuild p) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int s_dead;
    __shared__ int64_t s_w[GS_WARPS];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned full = 0xffffffffu;
    const int rank = blockIdx.x, blocks = gridDim.x;
    const int warp_id = rank + warp * blocks, warps = blocks * GS_WARPS;
    const int64_t nv = p.nv, gtid = (int64_t)rank * GS_THREADS + tid;
    const int64_t gthreads = (int64_t)blocks * GS_THREADS;
    unsigned round = 0;
    auto barrier = [&]() -> bool {
        const bool ok = all_blocks<GRID>(p.arrived, round, s_dead, p.polls);
        if (!ok && tid == 0) p.out->status = GS_TIMEOUT;
        return ok;
    };
    if (tid == 0) s_dead = 0;
    if (rank == 0 && tid < RS_CTL) p.ctl[tid] = 0;
    for (int64_t i = gtid; i < nv; i += gthreads) {
        p.first_ref[i] = INT_MAX;
        if (p.ref) p.first_pos[i] = INT_MAX;
        p.mcount[i] = 0;
        p.mfill[i] = 0;
        p.ecount[i] = 0;
    }
    if (!barrier()) return;
    // first member of each community, by reference id and by position
    for (int64_t i = gtid; i < nv; i += gthreads) {
        const int32_t c = p.comm[i];
        atomicMin(p.first_ref + c, vg_rid(p.ref, (int32_t)i));
        if (p.ref) atomicMin(p.first_pos + c, (int32_t)i);
    }
    if (!barrier()) return;
    // ranks of the first members: each block counts its slice, then numbers it
    const int64_t per = (nv + blocks - 1) / blocks;
    const int64_t lo = min(nv, rank * per), hi = min(nv, lo + per);
    auto heads_ref = [&](int64_t r) -> int { return __ldcg(p.first_ref + p.comm[pos_of(p.pos, r)]) == r; };
    auto heads_pos = [&](int64_t q) -> int { return __ldcg(p.first_pos + p.comm[q]) == q; };
    {
        int64_t a = 0, b = 0, total;
        for (int64_t i = lo + tid; i < hi; i += GS_THREADS) {
            a += heads_ref(i);
            if (p.ref) b += heads_pos(i);
        }
        block_excl(a, total, s_w);
        if (tid == 0) p.part[3 * rank] = total;
        block_excl(b, total, s_w);
        if (tid == 0) p.part[3 * rank + 1] = total;
    }
    if (!barrier()) return;
    const int64_t nc = block_prefix_of(p.part, blocks, s_w);
    {
        // the new numbers go to moff (by reference id) and mbase (by position) first: the
        // first-member arrays are still read by the other blocks
        int64_t run = block_prefix_of(p.part, rank, s_w), total;
        for (int64_t t = lo; t < hi; t += GS_THREADS) {
            const int64_t i = t + tid;
            const int h = i < hi ? heads_ref(i) : 0;
            const int64_t e = block_excl(h, total, s_w);
            if (h) p.moff[i] = run + e;
            run += total;
        }
        if (p.ref) {
            run = block_prefix_of(p.part + 1, rank, s_w);
            for (int64_t t = lo; t < hi; t += GS_THREADS) {
                const int64_t i = t + tid;
                const int h = i < hi ? heads_pos(i) : 0;
                const int64_t e = block_excl(h, total, s_w);
                if (h) p.mbase[i] = run + e;
                run += total;
            }
        }
    }
    if (!barrier()) return;
    for (int64_t c = gtid; c < nv; c += gthreads) {
        const int32_t fr = __ldcg(p.first_ref + c);
        if (fr == INT_MAX) continue;
        const int32_t nr = (int32_t)__ldcg(p.moff + fr);
        p.first_ref[c] = nr;
        if (p.ref) {
            const int32_t np = (int32_t)__ldcg(p.mbase + __ldcg(p.first_pos + c));
            p.first_pos[c] = np;
            p.next_ref[np] = nr;
            p.next_pos[nr] = np;
        }
    }
    if (!barrier()) return;
    // row (position) and key (reference id) of a community in the next level
    const int32_t *row_of = p.ref ? p.first_pos : p.first_ref, *key_of = p.first_ref;
    for (int64_t i = gtid; i < nv; i += gthreads) {
        const int32_t row = __ldcg(row_of + p.comm[i]);
        atomicAdd(p.mcount + row, 1);
        atomicAdd((unsigned long long *)p.ecount + row,
                  (unsigned long long)(p.rowptr[i + 1] - p.rowptr[i]));
    }
    if (!barrier()) return;
    // where each row's members and entries start; rows and segments a block takes
    const int64_t rper = (nc + blocks - 1) / blocks;
    const int64_t rlo = min(nc, rank * rper), rhi = min(nc, rlo + rper);
    {
        int64_t a = 0, b = 0, total;
        for (int64_t r = rlo + tid; r < rhi; r += GS_THREADS) {
            a += __ldcg(p.mcount + r);
            b += __ldcg(p.ecount + r);
        }
        block_excl(a, total, s_w);
        if (tid == 0) p.part[3 * rank] = total;
        block_excl(b, total, s_w);
        if (tid == 0) p.part[3 * rank + 1] = total;
    }
    if (!barrier()) return;
    {
        int64_t ma = block_prefix_of(p.part, rank, s_w), ea = block_prefix_of(p.part + 1, rank, s_w);
        for (int64_t t = rlo; t < rhi; t += GS_THREADS) {
            const int64_t r = t + tid;
            const int64_t m = r < rhi ? __ldcg(p.mcount + r) : 0, e = r < rhi ? __ldcg(p.ecount + r) : 0;
            int64_t mt, et;
            const int64_t mp = block_excl(m, mt, s_w), ep = block_excl(e, et, s_w);
            if (r < rhi) {
                p.mbase[r] = ma + mp;
                p.rstart[r] = ea + ep;
                if (m > 32) p.biglist[atomicAdd(p.ctl + RS_BIG_ROWS, 1)] = (int32_t)r;
                const int64_t reads = e > SmallBlockTable::MAXU
                                          ? (nc + SmallBlockTable::MAXU - 1) / SmallBlockTable::MAXU
                                          : 1;
                if (e * reads > rs_max_reads(p.integral, reads)) p.ctl[RS_REFUSED] = 1;
                if (e > RS_BIG_L) p.longlist[atomicAdd(p.ctl + RS_LONG_SEGS, 1)] = (int32_t)r;
            }
            ma += mt;
            ea += et;
        }
    }
    if (!barrier()) return;
    if (__ldcg(p.ctl + RS_REFUSED)) { // the same in every block
        if (rank == 0 && tid == 0) p.out->status = GS_REFUSED;
        return;
    }
    for (int64_t i = gtid; i < nv; i += gthreads) {
        const int32_t row = __ldcg(row_of + p.comm[i]);
        p.mlist[__ldcg(p.mbase + row) + atomicAdd(p.mfill + row, 1)] = vg_rid(p.ref, (int32_t)i);
    }
    if (!barrier()) return;
    // each row's members in reference order, replaced by their positions, and where each
    // one's entries go
    for (int64_t r = warp_id; r < nc; r += warps) {
        const int m = __ldcg(p.mcount + r);
        if (m > 32) continue;
        const int64_t base = __ldcg(p.mbase + r);
        int32_t x = lane < m ? __ldcg(p.mlist + base + lane) : INT_MAX;
        if (m > 1) {
#pragma unroll
            for (int k = 2; k <= 32; k <<= 1)
#pragma unroll
                for (int j = k >> 1; j > 0; j >>= 1) {
                    const int32_t y = __shfl_xor_sync(full, x, j);
                    const bool up = (lane & k) == 0, low = (lane & j) == 0;
                    x = low == up ? min(x, y) : max(x, y);
                }
        }
        int64_t d = 0, total;
        int32_t q = 0;
        if (lane < m) {
            q = pos_of(p.pos, x);
            d = p.rowptr[q + 1] - p.rowptr[q];
        }
        const int64_t o = warp_excl(d, total);
        if (lane < m) {
            p.mlist[base + lane] = q;
            p.moff[base + lane] = __ldcg(p.rstart + r) + o;
        }
    }
    const int nbig = __ldcg(p.ctl + RS_BIG_ROWS);
    for (int b = rank; b < nbig; b += blocks) { // uniform over the block
        uint32_t *bits = reinterpret_cast<uint32_t *>(smem_raw);
        const int words = (int)((nv + 31) / 32), each = (words + GS_THREADS - 1) / GS_THREADS;
        const int64_t r = __ldcg(p.biglist + b);
        const int64_t base = __ldcg(p.mbase + r), m = __ldcg(p.mcount + r);
        __syncthreads();
        for (int i = tid; i < words; i += GS_THREADS) bits[i] = 0;
        __syncthreads();
        for (int64_t k = tid; k < m; k += GS_THREADS) {
            const int32_t x = __ldcg(p.mlist + base + k);
            atomicOr(bits + (x >> 5), 1u << (x & 31));
        }
        __syncthreads();
        int64_t cnt = 0, total;
        const int w0 = min(words, tid * each), w1 = min(words, w0 + each);
        for (int i = w0; i < w1; i++) cnt += __popc(bits[i]);
        int64_t at = base + block_excl(cnt, total, s_w);
        for (int i = w0; i < w1; i++)
            for (uint32_t y = bits[i]; y; y &= y - 1) p.mlist[at++] = pos_of(p.pos, i * 32 + __ffs(y) - 1);
        __syncthreads();
        int64_t run = __ldcg(p.rstart + r);
        for (int64_t t = 0; t < m; t += GS_THREADS) {
            const int64_t k = t + tid;
            int64_t d = 0;
            if (k < m) {
                const int32_t q = __ldcg(p.mlist + base + k);
                d = p.rowptr[q + 1] - p.rowptr[q];
            }
            const int64_t o = block_excl(d, total, s_w);
            if (k < m) p.moff[base + k] = run + o;
            run += total;
        }
    }
    if (!barrier()) return;
    // entries to their segments, neighbours as keys: eight lanes per member, a warp when
    // rows average 64 entries
    {
        const int g = p.ne >= 64 * nv ? 32 : 8, sub = tid & (g - 1);
        for (int64_t k = gtid / g; k < nv; k += gthreads / g) {
            const int32_t q = __ldcg(p.mlist + k);
            const int64_t o = __ldcg(p.moff + k), e0 = p.rowptr[q], len = p.rowptr[q + 1] - e0;
            for (int64_t j = sub; j < len; j += 4 * g) {
                int32_t t[4];
                double w[4];
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const int64_t i = j + u * g;
                    t[u] = i < len ? p.tail[e0 + i] : -1;
                    w[u] = i < len ? p.weight[e0 + i] : 0.0;
                }
#pragma unroll
                for (int u = 0; u < 4; u++)
                    if (t[u] >= 0) t[u] = __ldcg(key_of + p.comm[t[u]]);
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const int64_t i = j + u * g;
                    if (i < len) {
                        p.gk[o + i] = t[u];
                        p.gw[o + i] = w[u];
                    }
                }
            }
        }
    }
    if (!barrier()) return;
    {
        SmallWarpTable &S = reinterpret_cast<SmallWarpTable *>(smem_raw)[warp];
        for (int64_t r = warp_id; r < nc; r += warps) {
            const int64_t L = __ldcg(p.ecount + r);
            if (L > RS_BIG_L) continue;
            const int U = warp_segment<true>(S, __ldcg(p.rstart + r), L, p.gk, p.gw, p.uk, p.uw, true);
            if (lane == 0) {
                if (U >= 0)
                    p.ucount[r] = U;
                else
                    p.longlist[atomicAdd(p.ctl + RS_LONG_SEGS, 1)] = (int32_t)r;
            }
            __syncwarp();
        }
    }
    if (!barrier()) return;
    // the other segments, a block each
    const int nlong = __ldcg(p.ctl + RS_LONG_SEGS);
    for (int b = rank; b < nlong; b += blocks) { // uniform over the block
        const int64_t r = __ldcg(p.longlist + b);
        SmallBlockTable &T = *reinterpret_cast<SmallBlockTable *>(smem_raw);
        const int64_t s0 = __ldcg(p.rstart + r), L = __ldcg(p.ecount + r);
        int64_t U = block_segment<true>(T, s0, L, p.integral, p.gk, p.gw, p.uk, p.uw, s0);
        if (U < 0) { // more keys than the table takes: a range of as many key values at a time
            U = 0;
            for (int64_t lo = 0; lo < nc; lo += SmallBlockTable::MAXU)
                U += block_segment<true>(T, s0, L, p.integral, p.gk, p.gw, p.uk, p.uw, s0 + U,
                                         (int32_t)lo, (int32_t)(lo + SmallBlockTable::MAXU));
        }
        if (tid == 0) p.ucount[r] = U;
    }
    if (!barrier()) return;
    // the next level's row offsets
    {
        int64_t a = 0, total;
        int32_t most = 0;
        for (int64_t r = rlo + tid; r < rhi; r += GS_THREADS) {
            const int64_t u = __ldcg(p.ucount + r);
            a += u;
            most = max(most, (int32_t)u);
        }
        __syncwarp();
        vg_raise(p.ctl + RS_LONGEST, most);
        block_excl(a, total, s_w);
        if (tid == 0) p.part[3 * rank + 2] = total;
    }
    if (!barrier()) return;
    {
        int64_t run = block_prefix_of(p.part + 2, rank, s_w), total;
        for (int64_t t = rlo; t < rhi; t += GS_THREADS) {
            const int64_t r = t + tid;
            const int64_t e = block_excl(r < rhi ? __ldcg(p.ucount + r) : 0, total, s_w);
            if (r < rhi) p.rowptr_out[r] = run + e;
            run += total;
        }
        if (rank == blocks - 1 && tid == 0) {
            p.rowptr_out[nc] = run;
            p.out->nc = nc;
            p.out->m = run;
            p.out->longest = __ldcg(p.ctl + RS_LONGEST);
        }
    }
}

// the next level into arrays of its own size: G lanes per row
template <int G>
__global__ void k_rebuild_small_copy(SmallRebuild p, int64_t nc, int64_t *__restrict__ rowptr,
                                     int32_t *__restrict__ tail, double *__restrict__ w,
                                     int32_t *__restrict__ ref, int32_t *__restrict__ pos) {
    const int sub = threadIdx.x & (G - 1);
    const int64_t grp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / G;
    const int64_t ng = ((int64_t)gridDim.x * blockDim.x) / G;
    for (int64_t r = grp; r <= nc; r += ng) {
        const int64_t o = p.rowptr_out[r];
        if (sub == 0) rowptr[r] = o;
        if (r == nc) break;
        if (sub == 0 && ref) {
            ref[r] = p.next_ref[r];
            pos[r] = p.next_pos[r];
        }
        const int64_t s = p.rstart[r], len = p.rowptr_out[r + 1] - o;
        for (int64_t j = sub; j < len; j += G) {
            const int32_t k = p.uk[s + j];
            tail[o + j] = ref ? p.next_pos[k] : k;
            w[o + j] = p.uw[s + j];
        }
    }
}

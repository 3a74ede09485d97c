// A whole Louvain phase of a small graph in one launch (included by louvain.cu).
//
// What bounds a small phase is not memory: with one launch per step, an iteration over a
// few thousand vertices waits for six launches and a read-back (30-70 us) while its sweep
// needs a few. Here one launch keeps the phase: degrees, 1/(2m), every sweep, the community
// update, the modularity and the loop test run between barriers, and the host waits once.
// The smallest graphs use one thread-block cluster (up to 16 blocks) and its hardware
// barrier; the others one block on every SM, launched cooperatively, with a barrier in
// global memory whose wait is bounded.
//
// Measured, phase by launches -> here (RGG and ER levels, vertices / entries): 1,201 / 8,082,
// 12 iterations 610 -> 186 us; 2,324 / 244,610, 5 iterations 751 -> 279 us; 31,145 / 250,126,
// 9 iterations 602 -> 282 us. Where the lines lie: a cluster takes up to 16,384 entries
// (170 / 881: 95 us with the whole grid, 101 with a cluster; 33 / 228: 61 and 49); the path
// ends at 2^21 entries because the rows of larger graphs fill the chip and the general
// sweeps stage them better (300,007 / 2.8e6: 1.49 ms by launches, 1.39 here; 348,203 / 6.5e6:
// 1.54 and 2.31). With at most four vertices per warp of the launch every row gets a warp:
// a thread's row of 32 entries is a 5-12 us chain, a warp's about 2 us.
//
// With colors a sweep and an update per color run the same way (30,000 / 479,846, 4
// iterations of a -c 8 phase: 1.97 -> 0.94 ms; 150,000 / 1.8e6 with hubs: 4.4 -> 2.7).
//
// The rows go through the same code as the general sweeps (thread_vertex, warp_vertex,
// cta_vertex), with loads that bypass the caches a previous iteration may have filled, and
// the sums keep the chunks and trees of k_seg_sum_* / k_apply_seg / k_mod_seg, so every
// result has the bits the general path gives (real weights: up to the order of the
// community updates' atomics, as between two runs of it).

constexpr int SP_THREADS = GS_THREADS;
constexpr int SP_WARPS = GS_WARPS;
constexpr int SP_T = 32;       // rows up to here: one thread each
constexpr int SP_CAP = 16384;  // slots of a block's table: rows of up to half as many communities
// entries of a row (of a multigraph: the others' rows have no more than their communities) up to
// which its one block is not waited for longer than launches would take: phases with one such
// row by launches and here, 20,000 entries 0.51 and 0.29 ms, 50,000 0.48 and 0.43, 80,000 0.53 and
// 0.69, 800,000 0.50 and 5.1
constexpr int64_t SP_MAX_ROW = 49152;
constexpr int SP_UNITS = SEG_CHUNK == 2048 && SEG_THREADS == 256 ? 8 : -1; // warps per chunk
#ifndef VG_SP_MAX_NV
#define VG_SP_MAX_NV VG_ONE_LAUNCH_NV
#endif
#ifndef VG_SP_MAX_NE
#define VG_SP_MAX_NE (1 << 21)
#endif
#ifndef VG_SP_NE_PER_CTA
#define VG_SP_NE_PER_CTA 1024 // entries a block gets before the cluster grows
#endif
#ifndef VG_SP_CLUSTER_NE
#define VG_SP_CLUSTER_NE 16384 // entries up to which a cluster takes the phase
#endif
#ifndef VG_SP_WARP_ROWS
#define VG_SP_WARP_ROWS 4 // vertices per warp up to which every row gets a warp
#endif
constexpr int64_t SP_MAX_NV = VG_SP_MAX_NV;
constexpr int64_t SP_MAX_NE = VG_SP_MAX_NE;
static_assert(SP_UNITS == 8, "the chunk sums below assume 2048-entry chunks of 256 threads");
static_assert(SP_MAX_NV <= (int64_t)SEG_FINAL * SEG_CHUNK && SEG_FINAL == 1024,
              "one chunk per thread of k_mod_seg's block in the final sums");

constexpr int SP_MAX_COLORS = 256;
// rows by length: a thread (or a warp, when they are few), a warp, a block
enum { ROW_SHORT, ROW_WARP, ROW_BLOCK, SP_CLASSES };
// the words of SmallPhase::ctl: rows per (color, class), then those placed so far
enum { CTL_REFUSED, CTL_NOPRUNE, CTL_COUNT };
__host__ __device__ constexpr int sp_ctl_words(int colors) { return CTL_COUNT + 2 * SP_CLASSES * colors; }

// what the kernel tells the host (pinned memory)
struct SmallOut {
    double mod;      // prevMod at the break
    double sweep_ns; // time between the barriers around the sweeps
    int32_t iters;
    int32_t status;  // GS_DONE; GS_REFUSED when a row may hold more communities than a block's
                     // table, or has more than SP_MAX_ROW entries
};

struct SmallPhase {
    LiveArgs a; // rowptr .. ne; constant, curr and target are set by the kernel
    int64_t nv;
    double *vdeg, *cdeg;
    int32_t *csize;
    int32_t *buf[3]; // past, curr, target at the start
    uint8_t *active;
    double *pa, *pb; // early termination 2 / 4
    double *part;    // 3 doubles per warp of each chunk
    int32_t *list;   // rows by (color, class); without colors only the long ones
    int32_t *ctl;    // sp_ctl_words(ncolors) words, zeroed by the first block
    int32_t *comm;   // the result
    double lower, threshold, one_minus_delta;
    int32_t et, integral;
    const int32_t *colors; // null: every vertex in one sweep; else a sweep and a community
                           // update per color (louvain.cpp:724-735)
    int32_t ncolors;       // uncolored (-1) vertices go with the last one
    unsigned *arrived; // (GRID) blocks that reached the grid's barriers so far (starts at 0)
    int32_t polls;     // of one wait there
    int32_t max_iters; // then the launch ends with GS_ENDLESS
    SmallOut *out;
};

__device__ __forceinline__ uint64_t global_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %globaltimer;\n" : "=l"(t));
    return t;
}

__device__ __forceinline__ double warp_tree(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = __dadd_rn(v, __shfl_down_sync(0xffffffffu, v, o));
    return v;
}

// The sums of all chunks from their warps' sums, x(q, w) that of warp w in chunk q: the
// trees of block_sum over a chunk's eight warps, then over SEG_FINAL threads, one chunk
// each. The whole block calls it; K sums at once, the result in s_sum[0..K).
template <int K, class X>
__device__ __forceinline__ void small_final(int64_t chunks, X x, double (*s_part)[32], double *s_sum) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int vw = warp; vw < SEG_FINAL / 32; vw += SP_WARPS) {
        const int q = vw * 32 + lane;
#pragma unroll
        for (int k = 0; k < K; k++) {
            double s = 0.0;
            if (vw * 32 < chunks) { // uniform over the warp
                if (q < chunks) {
                    double y[SP_UNITS];
#pragma unroll
                    for (int w = 0; w < SP_UNITS; w++) y[w] = x(q, w, k);
                    s = __dadd_rn(__dadd_rn(__dadd_rn(y[0], y[4]), __dadd_rn(y[2], y[6])),
                                  __dadd_rn(__dadd_rn(y[1], y[5]), __dadd_rn(y[3], y[7])));
                }
                s = warp_tree(s);
            }
            if (lane == 0) s_part[k][vw] = s;
        }
    }
    __syncthreads();
    if (warp < K) {
        const double s = warp_tree(s_part[warp][lane]);
        if (lane == 0) s_sum[warp] = s;
    }
    __syncthreads();
}

// vertex v (row at e0, degree d <= 32) by one warp, an entry per lane and no table: the
// lowest lane of each community folds its peers in lane order (the row's CSR order) and
// evaluates it, all communities' degrees in one gather. stage: 32 doubles of the warp's.
template <class A>
__device__ __forceinline__ void warp_short_vertex(const A &a, int32_t v, int64_t e0, int d, double cst,
                                                  double *stage) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    if (a.active && !A::ld(a.active + v)) {
        if (lane == 0) a.cw[v] = A::ld(a.frozen + v);
        return;
    }
    const int32_t cc = A::ld(a.curr + v);
    const double vd = A::ld(a.vdeg + v);
    const double ccDeg = A::ld(a.cdeg + cc);
    const bool has = lane < d;
    int32_t t = -1, c = -1;
    double w = 0.0, ay = 0.0;
    if (has) {
        t = a.tail[e0 + lane];
        w = a.weight[e0 + lane];
        c = A::ld(a.curr + t);
        ay = A::ld(a.cdeg + c);
    }
    stage[lane] = w;
    const unsigned peers = __match_any_sync(full, has ? c : (-1 - lane));
    __syncwarp();
    const bool leader = has && lane == __ffs(peers) - 1;
    const unsigned above = leader ? peers & ~((2u << lane) - 1u) : 0u;
    w = vg_fold_peers(w, stage, above, __reduce_max_sync(full, (unsigned)__popc(above)));
    double selfLoop = 0.0;
    for (unsigned m = __ballot_sync(full, has && t == v); m; m &= m - 1)
        selfLoop = __dadd_rn(selfLoop, stage[__ffs(m) - 1]);
    const unsigned own = __ballot_sync(full, leader && c == cc);
    const double at_own = __shfl_sync(full, w, own ? __ffs(own) - 1 : 0);
    const double counter0 = own ? at_own : 0.0;
    const double eix = __dsub_rn(counter0, selfLoop);
    const double ax = __dsub_rn(ccDeg, vd);
    double gain = 0.0;
    int32_t cand = INT_MAX;
    bool ok = false;
    if (leader && c != cc) {
        const double g = gain_of(w, eix, vd, ay, ax, cst);
        if (g > 0.0) {
            ok = true;
            gain = g;
            cand = c;
        }
    }
    warp_argbest(ok, gain, cand, a.ref);
    if (lane == 0) {
        int32_t ccSize, csz;
        sizes_for_rule(a, ok, cand, cc, ccSize, csz);
        commit_vertex(a, v, cc, ccSize, vd, d > 0, counter0, ok, cand, csz);
    }
    __syncwarp();
}

// dynamic shared memory: the rows' slots and tables, one class at a time
constexpr size_t SP_WORK_BYTES = warp_smem_bytes<WT_CAP, SP_WARPS>();
static_assert(SP_WORK_BYTES >= sizeof(double) * SP_T * SP_THREADS &&
                  SP_WORK_BYTES >= cta_smem_bytes(SP_CAP, SP_THREADS) &&
                  SP_WORK_BYTES >= sizeof(double) * 2 * VG_FOLD_STEP * SP_WARPS,
              "every class's tables must fit the block's work area");

template <bool GRID>
__global__ void __launch_bounds__(SP_THREADS, 1) k_phase_small(SmallPhase p) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ CtaShared<SP_THREADS> sh;
    __shared__ int s_dead, s_base[SP_CLASSES * SP_MAX_COLORS + 1];
    __shared__ int64_t s_w[SP_WARPS];
    __shared__ double s_sum[3], s_part[3][32];
    double *work = reinterpret_cast<double *>(smem_raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rank = blockIdx.x, blocks = gridDim.x; // without GRID the grid is one cluster
    unsigned round = 0;
    auto barrier = [&]() -> bool {
        const bool ok = all_blocks<GRID>(p.arrived, round, s_dead, p.polls);
        if (!ok && tid == 0) p.out->status = GS_TIMEOUT;
        return ok;
    };
    const int64_t nv = p.nv;
    const int64_t chunks = (nv + SEG_CHUNK - 1) / SEG_CHUNK;
    LiveArgs a = p.a;

    const int warp_id = rank + warp * blocks, warps = blocks * SP_WARPS; // neighbours on other SMs

    if (tid == 0) s_dead = 0;
    const int buckets = SP_CLASSES * p.ncolors;
    int32_t *count = p.ctl + CTL_COUNT, *placed = count + buckets;
    if (rank == 0)
        for (int i = tid; i < sp_ctl_words(p.ncolors); i += SP_THREADS) p.ctl[i] = 0;
    if (!barrier()) return;
    // Short rows' degrees are folded at once. The other rows (with colors: all) are counted
    // by color and class, then listed, so that a class spreads over the blocks wherever its
    // rows lie (a coarse level's longest rows are its first ones).
    auto bucket_of = [&](int64_t v, int64_t d) {
        const int cls = d <= SP_T ? ROW_SHORT : d <= WT_MAXDEG ? ROW_WARP : ROW_BLOCK;
        if (!p.colors) return cls == ROW_SHORT ? -1 : cls;
        const int32_t c = __ldg(p.colors + v);
        return (c < 0 ? p.ncolors - 1 : c) * SP_CLASSES + cls;
    };
    for (int64_t b = warp_id; b * 32 < nv; b += warps) {
        const int64_t v = b * 32 + lane;
        int bucket = -1;
        if (v < nv) {
            const int64_t e0 = a.rowptr[v], e1 = a.rowptr[v + 1];
            const int64_t d = e1 - e0;
            if (d <= SP_T) p.vdeg[v] = row_fold(a.weight, e0, e1);
            if (d > SP_MAX_ROW || min(d, nv) > SP_CAP / 2) p.ctl[CTL_REFUSED] = 1;
            bucket = bucket_of(v, d);
        }
        const unsigned peers = __match_any_sync(0xffffffffu, bucket);
        if (bucket >= 0 && lane == __ffs(peers) - 1) atomicAdd(count + bucket, __popc(peers));
    }
    if (!barrier()) return;
    if (__ldcg(p.ctl + CTL_REFUSED)) { // the same in every block
        if (rank == 0 && tid == 0) p.out->status = GS_REFUSED;
        return;
    }
    int rows = 0; // listed
    for (int t = 0; t < buckets; t += SP_THREADS) {
        int64_t total;
        const int64_t e = block_excl(t + tid < buckets ? __ldcg(count + t + tid) : 0, total, s_w);
        if (t + tid < buckets) s_base[t + tid] = rows + (int)e;
        rows += (int)total;
    }
    if (tid == 0) s_base[buckets] = rows;
    __syncthreads();
    for (int64_t b = warp_id; b * 32 < nv; b += warps) {
        const int64_t v = b * 32 + lane;
        const int bucket = v < nv ? bucket_of(v, a.rowptr[v + 1] - a.rowptr[v]) : -1;
        const unsigned peers = __match_any_sync(0xffffffffu, bucket);
        const int lead = __ffs(peers) - 1;
        int at = 0;
        if (bucket >= 0 && lane == lead) at = atomicAdd(placed + bucket, __popc(peers));
        at = __shfl_sync(0xffffffffu, at, lead);
        if (bucket >= 0) p.list[s_base[bucket] + at + __popc(peers & ((1u << lane) - 1u))] = (int32_t)v;
    }
    if (!barrier()) return;
    for (int i = warp_id; i < rows; i += warps) {
        const int32_t v = __ldcg(p.list + i);
        const int64_t E0 = a.rowptr[v], E1 = a.rowptr[v + 1];
        if (E1 - E0 <= SP_T) continue;
        double s = 0.0;
        if (p.integral) { // exact in any order
            for (int64_t k = E0 + lane; k < E1; k += 32) s = __dadd_rn(s, a.weight[k]);
            s = warp_tree(s);
        } else {
            const double *__restrict__ w = a.weight + E0;
            s = vg_warp_fold(E1 - E0, [w](int64_t j) { return w[j]; },
                                     work + (size_t)warp * 2 * VG_FOLD_STEP, 0.0, false);
        }
        if (lane == 0) p.vdeg[v] = s;
    }
    if (!barrier()) return;
    for (int64_t i = (int64_t)rank * SP_THREADS + tid; i < nv; i += (int64_t)blocks * SP_THREADS) {
        const double vd = __ldcg(p.vdeg + i);
        if (!(vd >= 0.0)) p.ctl[CTL_NOPRUNE] = 1;
        p.cdeg[i] = vd;
        p.csize[i] = 1;
        CommInfo z;
        z.deg = 0.0;
        z.size = 0;
        z.pad = 0;
        a.cupd[i] = z;
        for (int k = 0; k < 3; k++) p.buf[k][i] = (int32_t)i;
        if (p.active) p.active[i] = 1;
        if (p.pa) p.pa[i] = 0.0;
        if (p.pb) p.pb[i] = 1.0;
    }
    // 2m
    const int64_t units = chunks * SP_UNITS;
    for (int64_t u = warp_id; u < units; u += warps) {
        const int64_t lo = (u / SP_UNITS) * SEG_CHUNK, hi = min(lo + SEG_CHUNK, nv);
        double s = 0.0;
        for (int64_t i = lo + (u % SP_UNITS) * 32 + lane; i < hi; i += SEG_THREADS)
            s = __dadd_rn(s, __ldcg(p.vdeg + i));
        s = warp_tree(s);
        if (lane == 0) p.part[3 * u] = s;
    }
    if (!barrier()) return;
    small_final<1>(chunks, [&](int q, int w, int k) {
        return __ldcg(p.part + 3 * (q * SP_UNITS + w) + k);
    }, s_part, s_sum);
    const double cst = __ddiv_rn(1.0, s_sum[0]); // distCalcConstantForSecondTerm
    a.constant = cst;
    // no block overwrites p.part before the next barrier

    // community update and, with sums, those of the modularity (k_apply_seg)
    auto apply = [&](bool sums) {
        for (int64_t u = warp_id; u < units; u += warps) {
            const int64_t lo = (u / SP_UNITS) * SEG_CHUNK, hi = min(lo + SEG_CHUNK, nv);
            double le = 0.0, la2 = 0.0, frozen = 0.0;
            for (int64_t i = lo + (u % SP_UNITS) * 32 + lane; i < hi; i += SEG_THREADS) {
                const int4 raw = __ldcg(reinterpret_cast<const int4 *>(a.cupd + i));
                const double udeg = __hiloint2double(raw.y, raw.x);
                double cd = __ldcg(p.cdeg + i);
                if (raw.z != 0 || udeg != 0.0) {
                    cd = __dadd_rn(cd, udeg);
                    p.cdeg[i] = cd;
                    const int32_t ns = __ldcg(p.csize + i) + raw.z;
                    p.csize[i] = ns;
                    if (ns > 0 && !(cd >= 0.0)) p.ctl[CTL_NOPRUNE] = 1;
                    CommInfo z;
                    z.deg = 0.0;
                    z.size = 0;
                    z.pad = 0;
                    a.cupd[i] = z;
                }
                if (!sums) continue;
                le = __dadd_rn(le, __ldcg(a.cw + i));
                la2 = __dadd_rn(la2, __dmul_rn(cd, cd));
                if (p.active && !__ldcg(p.active + i)) frozen += 1.0;
            }
            if (!sums) continue;
            le = warp_tree(le);
            la2 = warp_tree(la2);
            frozen = warp_tree(frozen);
            if (lane == 0) {
                p.part[3 * u] = le;
                p.part[3 * u + 1] = la2;
                p.part[3 * u + 2] = frozen;
            }
        }
    };

    int ip = 0; // buf[ip], buf[ip + 1], buf[ip + 2] (mod 3): past, curr, target
    double *pcurr = p.pa, *pprev = p.pb;
    double prev = p.lower, sweep_ns = 0.0;
    int iters = 0;
    for (;;) {
        if (iters == p.max_iters) { // the same in every block
            if (rank == 0 && tid == 0) p.out->status = GS_ENDLESS;
            return;
        }
        iters++;
        int32_t *past = p.buf[ip], *curr = p.buf[(ip + 1) % 3], *target = p.buf[(ip + 2) % 3];
        a.curr = curr;
        a.target = target;
        const uint64_t t0 = rank == 0 && tid == 0 ? global_ns() : 0;
        for (int color = 0; color < p.ncolors; color++) {
            if (color) {
                if (!barrier()) return;
                apply(false); // the last color's update has the sums
                if (!barrier()) return;
            }
            // item i of the list goes to the block (warp) i modulo their number, so that the
            // colors' rows fall to different ones
            const int *base = s_base + SP_CLASSES * color;
            auto first = [](int from, int id, int n) { // smallest i >= from, i = id modulo n
                if (from <= id) return id;
                const int d = (from - id) % n;
                return d ? from + n - d : from;
            };
            int i = first(base[ROW_BLOCK], rank, blocks);
            if (i < base[SP_CLASSES]) { // uniform over the block
                const Table t = cta_table<SP_THREADS>(smem_raw, SP_CAP, sh);
                for (; i < base[SP_CLASSES]; i += blocks) {
                    const int32_t v = __ldcg(p.list + i);
                    const int64_t e0 = a.rowptr[v], d = a.rowptr[v + 1] - e0;
                    cta_vertex<SP_THREADS>(a, v, e0, d, min(d, nv), cst, t, sh);
                }
                __syncthreads();
            }
            // short rows: all vertices in turn, or the color's list
            const int s0 = p.colors ? base[ROW_SHORT] : 0;
            const int s1 = p.colors ? base[ROW_WARP] : (int)nv;
            const bool by_thread = s1 - s0 > VG_SP_WARP_ROWS * warps;
            if (by_thread) {
                for (int b = first(s0 / 32, warp_id, warps); b * 32 < s1; b += warps) {
                    const int i = b * 32 + lane;
                    if (i < s0 || i >= s1) continue;
                    const int32_t v = p.colors ? __ldcg(p.list + i) : i;
                    const int64_t e0 = a.rowptr[v];
                    const int64_t d = a.rowptr[v + 1] - e0;
                    if (d <= SP_T) thread_vertex<SP_T, SP_THREADS>(a, v, e0, (int)d, cst, work + tid);
                }
                __syncthreads();
            }
            if (!by_thread) {
                for (int i = first(s0, warp_id, warps); i < s1; i += warps) {
                    const int32_t v = p.colors ? __ldcg(p.list + i) : i;
                    const int64_t e0 = a.rowptr[v];
                    const int64_t d = a.rowptr[v + 1] - e0;
                    if (d <= SP_T) warp_short_vertex(a, v, e0, (int)d, cst, work + warp * 32);
                }
            }
            if (base[ROW_WARP] < base[ROW_BLOCK]) {
                if (!by_thread) __syncthreads(); // the stages of the short rows
                const Table t = warp_table<WT_CAP, SP_WARPS>(smem_raw, warp);
                for (i = first(base[ROW_WARP], warp_id, warps); i < base[ROW_BLOCK]; i += warps)
                    warp_vertex(a, __ldcg(p.list + i), cst, t);
            }
        }
        if (!barrier()) return;
        if (rank == 0 && tid == 0) sweep_ns += (double)(global_ns() - t0);
        apply(true);
        if (!barrier()) return;
        small_final<3>(chunks, [&](int q, int w, int k) {
            return __ldcg(p.part + 3 * (q * SP_UNITS + w) + k);
        }, s_part, s_sum);
        // the loop test (louvain.cpp:112-121, 553-563), the same in every block
        const double m = fabs(__dsub_rn(__dmul_rn(s_sum[0], cst),
                                        __dmul_rn(__dmul_rn(s_sum[1], cst), cst)));
        if (p.et >= 3 && s_sum[2] >= 90.0) break; // ET_CUTOFF
        if (m != m || __dsub_rn(m, prev) < p.threshold) break;
        prev = m < p.lower ? p.lower : m;
        if (p.et == 0) {
            ip = (ip + 1) % 3;
            continue;
        }
        for (int64_t i = (int64_t)rank * SP_THREADS + tid; i < nv; i += (int64_t)blocks * SP_THREADS) {
            if (p.et == 1 || p.et == 3)
                swap_et13(i, iters, past, curr, target, p.active, a.ref);
            else
                swap_et24(i, iters, p.one_minus_delta, past, curr, target, p.active, pcurr, pprev);
        }
        double *t = pcurr;
        pcurr = pprev;
        pprev = t;
        if (!barrier()) return;
    }
    for (int64_t i = (int64_t)rank * SP_THREADS + tid; i < nv; i += (int64_t)blocks * SP_THREADS)
        p.comm[i] = __ldcg(p.buf[ip] + i);
    if (rank == 0 && tid == 0) {
        p.out->mod = prev;
        p.out->sweep_ns = sweep_ns;
        p.out->iters = iters;
    }
}

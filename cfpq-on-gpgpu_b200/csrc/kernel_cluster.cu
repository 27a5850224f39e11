// Small closures: the whole semi-naive fixpoint of one query of at most 1024
// vertices inside ONE thread-block cluster, matrices and deltas resident in the
// cluster's shared memory.
//
// Why: a closure of this size is a chain of short iterations.  In the persistent
// kernel every iteration is about ten dependent round trips through L2 (plan,
// item list, k-list, staging, merge, grid barrier), 10-14 us whatever the work.
// Here an iteration reads rows of other CTAs' shared memory directly and ends
// with one hardware cluster barrier: 2.2 us for a light one at n = 300 (1.5 of
// picking terms, reading and merging, 0.8 of publishing and barrier), 3.7 at n =
// 1024.  Whole query, host edges: balanced brackets at n = 300 371 -> 199 us, a
// sparse random CNF at n = 1000 746 -> 480, same-generation at n = 1024 189 -> 159.
// Past that the bound is the traffic between the CTAs: about 19 bytes per ns
// and SM for 128-byte rows.
//
// Layout: CTA `rank` of the 16 owns rows [rank R, rank R + R) of every matrix
// (R = 16, 32 or 64 rows: n <= 256, 512, 1024), row-major, T words a row, three
// copies: the current matrix and two deltas used alternately.  A delta row counts
// only while its bit is set in the delta's row mask; every CTA holds the masks
// of all rows (whoever finds new bits sets the row's bit in all 16 copies of the
// delta's mask, and each CTA adds those to its own copy of the matrix's:
// cluster_rows.cuh), so empty rows are never read and nothing is cleared between
// iterations.
//
// Iteration t: the rules with a non-empty delta are picked, and a warp takes 32 /
// kTp rows r of a head C, kTp lanes a row, a word per lane.  For every picked
// term of a rule C -> A B the group lists the bits k of row r of delta A (of A)
// whose row k of B (of delta B) is not empty and ORs those rows, four in flight,
// straight from the owners' shared memory.  One group owns a row of a head, so
// it merges with plain stores.  Reads of rows that their owner is writing see a
// subset of the final bits (bits only get set) and at least those of the
// iteration's start; new bits are in the next delta, as in the other loops.
// The rows that got new bits are collected per CTA and announced once per head.
//
// The cost of an iteration grows with the bits of the deltas (row by row, no
// tiles; a term that finds nothing in a row group costs about 0.1 us): when the next iteration would read more than leave_reads rows per
// CTA, the cluster writes matrices and deltas back and leaves; the persistent
// kernel goes on from there.  Everything a barrier waits for is decided from
// counts and masks that all CTAs hold alike between two barriers, also while one
// of them is an iteration ahead (cluster_rows.cuh), so all of them leave in the
// same iteration.  The cluster barrier is the kernel's only wait, and unlike the
// polled ones of the other kernels it has no limit: it ends because every warp
// of every CTA passes the same barriers in the same order, whatever the data.
#include "cluster_rows.cuh"
#include "launch.h"

namespace cfpq {

namespace {

constexpr uint32_t kCtas = 16;  // non-portable cluster size
constexpr uint32_t kThreads = 512;
constexpr uint32_t kWarps = kThreads / 32;
constexpr uint32_t kList = 512;  // row numbers listed per warp
constexpr uint32_t kFlight = 4;  // rows in flight per group
constexpr uint32_t kLong = 8;    // listed rows of one group above which all groups of the warp share its list
constexpr unsigned kFull = 0xffffffffu;

struct ClusterArgs {
    const MatSlot *slots;
    ClusterRules rules;
    uint32_t nm, n, T, log2r;
    IterState *st;
    QueryTrack qt;
    unsigned long long *phase_log;
    uint32_t phase_log_iters;
    uint32_t leave_reads;
    IterState *host_st;
    const uint32_t *flag_src;
    uint32_t *flag_dst;
};

__device__ __forceinline__ uint32_t map_rank(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ uint64_t ld_cluster(uint32_t addr) {
    uint64_t v;
    asm volatile("ld.shared::cluster.u64 %0, [%1];" : "=l"(v) : "r"(addr));
    return v;
}
// (32-bit: 64-bit OR reductions on another CTA's shared memory lost updates)
__device__ __forceinline__ void red_or_cluster(uint32_t addr, uint32_t v) {
    asm volatile("red.relaxed.cluster.shared::cluster.or.b32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ void red_add_cluster(uint32_t addr, uint32_t v) {
    asm volatile("red.relaxed.cluster.shared::cluster.add.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ void cluster_barrier() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Shared memory, in 64-bit words: current matrices, two deltas (nm * R * T
// each), row masks (three deltas' and the current matrices', nm * T each), row
// lists (kWarps * kList 16-bit row numbers), new-bit counts per matrix (3 * 32),
// this iteration's new rows and bits per head.
__host__ __device__ inline uint32_t cluster_words(uint32_t nm, uint32_t T, uint32_t log2r) {
    return 3 * nm * (T << log2r) + 4 * nm * T + kWarps * kList / 4 + 3 * 16 + 32 + 16;
}

// Position of the n-th (0-based) set bit of x (x has more than n set bits).
__device__ __forceinline__ uint32_t nth_set(uint32_t x, uint32_t n) {
    for (; n; --n) x &= x - 1;
    return __ffs(x) - 1;
}

template <uint32_t kTp>
__global__ void __launch_bounds__(kThreads, 1) k_closure_cluster(const __grid_constant__ ClusterArgs a) {
    extern __shared__ __align__(16) uint64_t sm[];
    constexpr uint32_t kGroups = 32 / kTp, kCap = kList / kGroups;  // rows per warp, list entries per row
    static_assert(kCap >= 64, "a word's bits fit a row's list");
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, rank = blockIdx.x;
    const uint32_t group = lane / kTp, sub = lane % kTp;
    const uint32_t nm = a.nm, T = a.T, log2r = a.log2r, R = 1u << log2r, n = a.n;
    const uint32_t mat = T << log2r;  // words of one matrix's rows
    uint64_t *const cur = sm, *const dlt = sm + (size_t)nm * mat, *const masks = dlt + 2 * (size_t)nm * mat,
                    *const behind = masks + 4 * nm * T;
    uint16_t *const lists = reinterpret_cast<uint16_t *>(behind) + warp * kList, *const list = lists + group * kCap;
    uint32_t *const cnt = reinterpret_cast<uint32_t *>(behind + kWarps * kList / 4);  // [3][32]
    const ClusterRows rows{masks, masks + 3 * nm * T, cnt, nm, T};
    uint32_t *const newrow = cnt + 96;   // [32][2]: rows of this CTA with new bits, per head
    uint32_t *const newbits = newrow + 64;  // [32]
    const uint32_t row0 = rank << log2r, mine = row0 < n ? min(R, n - row0) : 0u;

    for (uint32_t i = tid; i < 4 * nm * T; i += kThreads) masks[i] = 0;
    if (tid < 192) cnt[tid] = 0;  // and newrow, newbits
    cluster_barrier();  // every CTA's masks and counts are zero before anyone adds to them

    // rows of matrix m with new bits (two words of row bits, this CTA's rows)
    // and their number, into every CTA's masks and counts (one warp)
    auto publish = [&](uint32_t m, uint32_t buf, uint32_t lo, uint32_t hi, uint32_t add) {
        if (lane >= kCtas) return;
        rows.publish(buf, m, row0 >> 6, lo, hi, add,
                     [&](uint32_t *p, uint32_t v) { red_or_cluster(map_rank(smem_addr(p), lane), v); },
                     [&](uint32_t *p, uint32_t v) { red_add_cluster(map_rank(smem_addr(p), lane), v); });
    };
    // (one lane) rows `bits` (from row r on) of slot i have `add` new bits
    auto note = [&](uint32_t i, uint32_t r, uint32_t bits, uint32_t add) {
        const uint32_t at = (row0 + r) & 63;  // r is a multiple of kGroups: the bits stay in one word
        atomicOr(&newrow[2 * i + (at >> 5)], bits << (at & 31));
        atomicAdd(&newbits[i], add);
    };
    for (uint32_t i = tid; i < nm * mat; i += kThreads) {  // rows fastest: 8-byte neighbours in the tiles
        const uint32_t r = i & (R - 1), w = (i >> log2r) % T, m = (i >> log2r) / T;
        cur[((m << log2r) + r) * T + w] =
            r < mine ? a.slots[m].cur.bits[tile_offset(T, (row0 + r) >> 6, w) + ((row0 + r) & 63)] : 0ULL;
    }
    __syncthreads();
    const uint32_t rg = R / kGroups;  // row groups of a matrix
    auto group_bits = [&](bool on) {  // bit g: group g has a lane with `on`
        const unsigned bal = __ballot_sync(kFull, on);
        uint32_t bits = 0;
#pragma unroll
        for (uint32_t g = 0; g < kGroups; ++g)
            bits |= ((bal >> (g * kTp)) & (kTp == 32 ? kFull : (1u << (kTp & 31)) - 1)) ? 1u << g : 0u;
        return bits;
    };
    for (uint32_t u = warp; u < nm * rg; u += kWarps) {
        const uint32_t m = u / rg, r = (u % rg) * kGroups;
        const uint64_t v = sub < T ? cur[((m << log2r) + r + group) * T + sub] : 0ULL;
        const uint32_t bits = group_bits(v != 0), add = __reduce_add_sync(kFull, (uint32_t)__popcll(v));
        if (bits && lane == 0) note(m, r, bits, add);
    }
    __syncthreads();
    for (uint32_t m = warp; m < nm; m += kWarps)
        if (newbits[m]) publish(m, 0, newrow[2 * m], newrow[2 * m + 1], newbits[m]);
    __syncthreads();
    if (tid < 96) newrow[tid] = 0;
    cluster_barrier();

    // this lane's rules (lane and 32 + lane) and the rules of head `lane`
    uint32_t b1s[2], b2s[2];
#pragma unroll
    for (uint32_t h = 0; h < 2; ++h) {
        const uint32_t ru = h * 32 + lane;
        b1s[h] = ru < a.rules.nrules ? a.rules.body1[ru] : 0u;
        b2s[h] = ru < a.rules.nrules ? a.rules.body2[ru] : 0u;
    }
    auto rules_of = [&](uint32_t hi) {
        const uint32_t s0 = a.rules.start[hi], k = a.rules.start[hi + 1] - s0;
        return (k >= 64 ? ~0ULL : (1ULL << k) - 1) << s0;
    };
    const uint64_t my_rules = lane < a.rules.nheads ? rules_of(lane) : 0ULL;
    const uint32_t halves = a.rules.nrules > 32 ? 2u : 1u;
    const uint32_t limit = a.leave_reads * ((n + R - 1) >> log2r);
    const uint32_t t0 = a.st->iter, max_iter = a.st->max_iter;
    uint32_t fresh = lane < nm ? cnt[lane] : 0u;  // new bits of matrix `lane` in the last iteration (at first: all)
    uint32_t total = fresh;                       // its set bits
    unsigned long long reads = 0, products = 0;
    uint32_t items = 0, outw = 0, neww = 0;  // row groups done, non-zero and new words merged
    uint32_t last_iter = 0, t = t0;
    unsigned long long done_ns = 0;
    bool left = false, changed = false;
    for (;; ++t) {
        const uint32_t it = t - t0, rd = ClusterRows::read_buffer(it), wr = ClusterRows::write_buffer(it), par = it & 1;
        if (rank == 0 && tid == 0 && a.phase_log && it < a.phase_log_iters)
            a.phase_log[3 * it] = globaltimer_ns();
        rows.open(it, tid, kThreads);
        const uint64_t *const D = dlt + par * (size_t)nm * mat;
        uint64_t *const Dn = dlt + (par ^ 1) * (size_t)nm * mat;
        const uint64_t *const dm = rows.delta_rows(rd, 0);
        // the terms with a non-empty delta (iteration 0: A * B once, as the first
        // term), and the heads that have one
        uint64_t on0 = 0, on1 = 0;
#pragma unroll
        for (uint32_t h = 0; h < 2; ++h) {
            if (h >= halves) break;
            const bool in = h * 32 + lane < a.rules.nrules;
            const uint32_t f1 = __shfl_sync(kFull, fresh, b1s[h]), f2 = __shfl_sync(kFull, fresh, b2s[h]);
            on0 |= (uint64_t)__ballot_sync(kFull, in && f1 && (it || f2)) << (32 * h);
            on1 |= (uint64_t)__ballot_sync(kFull, in && it && f2) << (32 * h);
        }
        const unsigned hmask = __ballot_sync(kFull, ((on0 | on1) & my_rules) != 0);
        const uint32_t units = __popc(hmask) * rg;
        for (uint32_t u = warp; u < units; u += kWarps) {
            const uint32_t hi = nth_set(hmask, u / rg), r0 = (u % rg) * kGroups, r = r0 + group, row = row0 + r;
            if (r0 >= mine) continue;
            const bool valid = r < mine && sub < T;
            const uint32_t head = a.rules.head[hi], w = sub < T ? sub : 0u;
            uint64_t acc = 0;
            // OR of the rows k of Q (the CTAs' shared memory) for the bits k of
            // the group's row x (a word per lane)
            auto gather = [&](uint64_t x, const uint64_t *Q) {
                if (!__any_sync(kFull, x != 0)) return;
                const uint32_t base = smem_addr(Q) + 8 * w, c = __popcll(x);
                uint32_t pre = c;  // inclusive scan over the group
#pragma unroll
                for (uint32_t o = 1; o < kTp; o <<= 1) {
                    const uint32_t v = __shfl_up_sync(kFull, pre, o, kTp);
                    if (sub >= o) pre += v;
                }
                const uint32_t all = __shfl_sync(kFull, pre, kTp - 1, kTp);
                // rows whose bits do not fit the list go kCap / 64 words at a time
                const uint32_t step = __any_sync(kFull, all > kCap) ? kCap / 64 : kTp;
                for (uint32_t w0 = 0; w0 < T; w0 += step) {
                    const uint32_t before = w0 ? __shfl_sync(kFull, pre, w0 - 1, kTp) : 0u;
                    const uint32_t upto = __shfl_sync(kFull, pre, min(w0 + step, kTp) - 1, kTp);
                    if (sub >= w0 && sub < w0 + step) {
                        uint64_t y = x;
                        uint32_t at = pre - c - before;
                        while (y) {
                            list[at++] = (uint16_t)(sub * 64 + (__ffsll((long long)y) - 1));
                            y &= y - 1;
                        }
                    }
                    __syncwarp();
                    const uint32_t len = upto - before;
                    // entries first, first + every, ... of a list, kFlight in flight
                    auto read_rows = [&](const uint16_t *l, uint32_t n_l, uint32_t first, uint32_t every) {
                        uint64_t o = 0;
                        for (uint32_t i = first; i < n_l; i += kFlight * every) {
                            uint64_t v[kFlight];
#pragma unroll
                            for (uint32_t q = 0; q < kFlight; ++q) {
                                const uint32_t k = l[min(i + q * every, n_l - 1)];
                                v[q] = ld_cluster(map_rank(base + (k & (R - 1)) * T * 8, k >> log2r));
                            }
#pragma unroll
                            for (uint32_t q = 0; q < kFlight; ++q) o |= v[q];
                        }
                        return o;
                    };
                    if (!__any_sync(kFull, len > kLong)) {
                        acc |= read_rows(list, len, 0, 1);
                    } else {  // one row after the other, all groups on it
#pragma unroll
                        for (uint32_t g = 0; g < kGroups; ++g) {
                            const uint32_t n_g = __shfl_sync(kFull, len, g * kTp);
                            uint64_t o = read_rows(lists + g * kCap, n_g, group, kGroups);
#pragma unroll
                            for (uint32_t d = kTp; d < 32; d <<= 1) o |= __shfl_xor_sync(kFull, o, d);
                            if (g == group) acc |= o;
                        }
                    }
                    if (sub == 0) reads += len;
                    __syncwarp();
                }
            };
            for (uint64_t todo = (on0 | on1) & rules_of(hi); todo; todo &= todo - 1) {
                const uint32_t ru = __ffsll((long long)todo) - 1, b1 = a.rules.body1[ru], b2 = a.rules.body2[ru];
                if ((on0 >> ru) & 1u) {
                    const bool fresh = valid && (it == 0 || ((dm[b1 * T + (row >> 6)] >> (row & 63)) & 1u));
                    const uint64_t *const P = it == 0 ? cur : D;
                    gather(fresh ? P[((b1 << log2r) + r) * T + w] & rows.rows(rd, b2, w) : 0ULL, cur + (size_t)b2 * mat);
                }
                if ((on1 >> ru) & 1u)
                    gather(valid ? cur[((b1 << log2r) + r) * T + w] & dm[b2 * T + w] : 0ULL, D + (size_t)b2 * mat);
            }
            const size_t at = ((size_t)(head << log2r) + r) * T + w;
            const uint64_t old = valid ? cur[at] : 0ULL, nw = valid ? acc & ~old : 0ULL;
            const uint32_t bits = group_bits(nw != 0);
            ++items;
            outw += valid && acc != 0;
            neww += nw != 0;
            if (!bits) continue;
            if (nw) cur[at] = old | nw;
            if (valid && ((bits >> group) & 1u)) Dn[at] = nw;
            const uint32_t add = __reduce_add_sync(kFull, (uint32_t)__popcll(nw));
            if (lane == 0) note(hi, r0, bits, add);
        }
        if (rank == 0 && tid == 0 && a.phase_log && it < a.phase_log_iters)
            a.phase_log[3 * it + 1] = globaltimer_ns();
        __syncthreads();
        for (uint32_t i = warp; i < a.rules.nheads; i += kWarps) {
            if (!newbits[i]) continue;
            publish(a.rules.head[i], wr, newrow[2 * i], newrow[2 * i + 1], newbits[i]);
            __syncwarp();
            if (lane < 2) newrow[2 * i + lane] = 0;
            if (lane == 0) newbits[i] = 0;
        }
        cluster_barrier();

        // ---- decision, the same in every warp of the cluster ----
        fresh = lane < nm ? cnt[wr * 32 + lane] : 0u;
        changed = __any_sync(kFull, fresh != 0);
        total += fresh;
        if (rank == 0 && warp == 0) {
            products += __popcll(on0) + __popcll(on1);
            const unsigned long long now = globaltimer_ns();
            if (lane == 0 && a.phase_log && it < a.phase_log_iters) a.phase_log[3 * it + 2] = now;
            if (changed) {
                last_iter = t + 1;
                done_ns = now;
            }
        }
        if (!changed || (max_iter && t + 1 >= max_iter)) break;
        // rows the next iteration reads: at most the bits of delta A and the bits
        // of A, once per rule; if that is above the limit, those whose row of B
        // (of delta B) is not empty, taking rows and bits as independent
        uint32_t est = 0;
#pragma unroll
        for (uint32_t h = 0; h < 2; ++h) {
            if (h >= halves) break;
            const uint32_t f1 = __shfl_sync(kFull, fresh, b1s[h]), f2 = __shfl_sync(kFull, fresh, b2s[h]);
            const uint32_t n1 = __shfl_sync(kFull, total, b1s[h]);
            if (h * 32 + lane < a.rules.nrules) est += f1 + (f2 ? n1 : 0u);
        }
        if (__reduce_add_sync(kFull, est) > limit) {
            uint32_t nrows = 0, ndelta = 0;  // non-empty rows of matrix `lane` and of its delta
            if (lane < nm)
                for (uint32_t w = 0; w < T; ++w) {
                    nrows += __popcll(rows.rows(wr, lane, w));
                    ndelta += __popcll(rows.delta_rows(wr, lane)[w]);
                }
            est = 0;
#pragma unroll
            for (uint32_t h = 0; h < 2; ++h) {
                if (h >= halves) break;
                const uint32_t f1 = __shfl_sync(kFull, fresh, b1s[h]), n1 = __shfl_sync(kFull, total, b1s[h]);
                const uint32_t r2 = __shfl_sync(kFull, nrows, b2s[h]), d2 = __shfl_sync(kFull, ndelta, b2s[h]);
                if (h * 32 + lane < a.rules.nrules)
                    est += (uint32_t)(((float)f1 * (float)r2 + (float)n1 * (float)d2) / (float)n);
            }
            left = __reduce_add_sync(kFull, est) > limit;
        }
        if (left) break;
    }

    // ---- write back what changed (and, on leaving, the deltas) ----
    const uint32_t wr = ClusterRows::write_buffer(t - t0), par = (t - t0) & 1;
    auto put = [&](const DevMat &m, const uint64_t *src, uint32_t r, uint32_t w, bool valid) {
        const uint32_t row = row0 + r, ti = row0 >> 6;  // R divides 64: the CTA's rows lie in one tile-row
        uint32_t add = 0;
        if (valid) {
            uint64_t *const dst = m.bits + tile_offset(T, ti, w) + (row & 63);
            const uint64_t v = src[r * T + w], nw = v & ~*dst;
            if (nw) *dst = v;
            add = (uint32_t)__popcll(nw);
        }
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) add += __shfl_xor_sync(kFull, add, o);
        if (R >= 32) add += __shfl_xor_sync(kFull, add, 16);  // else a half-warp holds a tile's rows
        if (add && (lane == 0 || (R < 32 && lane == 16))) {
            atomicAdd(m.nnz + (size_t)ti * T + w, add);
            atomicOr(m.occ + (size_t)ti * m.ow + (w >> 5), 1u << (w & 31));
        }
    };
    const uint32_t words = a.rules.nheads * mat;  // a multiple of 16 words: whole half-warps
    for (uint32_t i0 = warp * 32; i0 < words; i0 += kThreads) {
        const uint32_t i = i0 + lane;
        const bool in = i < words;
        const uint32_t r = i & (R - 1), w = in ? (i >> log2r) % T : 0u, head = a.rules.head[in ? (i >> log2r) / T : 0u];
        put(a.slots[head].cur, cur + (size_t)head * mat, r, w, in && r < mine);
        if (left) {
            const uint32_t row = row0 + r;
            const bool fresh = in && r < mine && ((rows.delta_rows(wr, head)[row >> 6] >> (row & 63)) & 1u);
            put(a.slots[head].dlt[(t + 1) & 1], dlt + ((par ^ 1) * (size_t)nm + head) * mat, r, w, fresh);
        }
    }
    for (int o = 16; o > 0; o >>= 1) reads += __shfl_xor_sync(kFull, reads, o);
    outw = __reduce_add_sync(kFull, outw);
    neww = __reduce_add_sync(kFull, neww);
    // per CTA first, in the row collectors (all zero now): an atomic of every warp
    // on the state's words took 6 us
    unsigned long long *const sum = reinterpret_cast<unsigned long long *>(newrow);
    const unsigned long long mine_sum = lane == 0 ? items : lane == 1 ? reads : lane == 2 ? outw : neww;
    if (lane < 4 && mine_sum) atomicAdd(sum + lane, mine_sum);
    __syncthreads();
    if (tid < 5 && sum[tid ? tid - 1 : 0]) {
        unsigned long long *const to = tid == 0   ? &a.st->items_by_variant[2]
                                       : tid == 1 ? &a.st->items_total
                                       : tid == 2 ? &a.st->tile_triples  // rows read until the end
                                       : tid == 3 ? &a.st->out_words
                                                  : &a.st->new_words;
        atomicAdd(to, sum[tid ? tid - 1 : 0]);
    }
    cluster_barrier();  // every CTA's counters are in, and no CTA's shared memory is read any more
    if (rank == 0 && tid == 0) {
        IterState *const st = a.st;
        // the rows read, of 64 T bit pairs each
        st->tile_triples = *(volatile unsigned long long *)&st->tile_triples * T / 4096;
        st->bytes_staged += (unsigned long long)nm * n * T * 8;
        st->products += products;
        st->dense_bitops += products * (unsigned long long)n * n * n;
        st->last_changed = changed;
        st->iter = t + 1;
        st->active = left;
        st->left = left;
        if (a.qt.last_iter && last_iter) {
            a.qt.last_iter[0] = last_iter;
            a.qt.done_ns[0] = done_ns;
        }
        __threadfence();
    }
    __syncthreads();
    if (rank == 0 && a.host_st) {
        const uint32_t *src = reinterpret_cast<const uint32_t *>(a.st);
        uint32_t *dst = reinterpret_cast<uint32_t *>(a.host_st);
        for (uint32_t i = tid; i < sizeof(IterState) / 4; i += kThreads) dst[i] = __ldcg(src + i);
        if (tid == 0 && a.flag_src) *a.flag_dst = __ldcg(a.flag_src);
    }
}

constexpr uint32_t kMaxSmem = 226 * 1024;

template <uint32_t kTp>
cudaError_t configure() {
    cudaError_t e = cudaFuncSetAttribute(k_closure_cluster<kTp>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(k_closure_cluster<kTp>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSmem);
}

void cluster_config(cudaLaunchConfig_t *cfg, cudaLaunchAttribute *attr, size_t smem, cudaStream_t s) {
    *cfg = cudaLaunchConfig_t{};
    cfg->gridDim = dim3(kCtas);
    cfg->blockDim = dim3(kThreads);
    cfg->dynamicSmemBytes = smem;
    cfg->stream = s;
    attr->id = cudaLaunchAttributeClusterDimension;
    attr->val.clusterDim.x = kCtas;
    attr->val.clusterDim.y = attr->val.clusterDim.z = 1;
    cfg->attrs = attr;
    cfg->numAttrs = 1;
}

uint32_t rows_log2(uint32_t n) { return n <= 256 ? 4 : n <= 512 ? 5 : 6; }

}  // namespace

int cluster_closure_available() {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr;
    cluster_config(&cfg, &attr, kMaxSmem, nullptr);
    int nc = 0;
    if (configure<4>() != cudaSuccess || configure<8>() != cudaSuccess || configure<16>() != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&nc, k_closure_cluster<16>, &cfg) != cudaSuccess)
        nc = 0;
    (void)cudaGetLastError();
    return nc > 0;
}

bool cluster_closure_fits(uint32_t nmats, size_t nrules, uint32_t n) {
    return n > 0 && n <= 64 * kCtas && nmats <= ClusterRules::kMats && nrules <= ClusterRules::kRules &&
           (size_t)cluster_words(nmats, (n + 63) / 64, rows_log2(n)) * 8 <= kMaxSmem;
}

cudaError_t launch_closure_cluster(const MatSlot *slots, uint32_t nmats, uint32_t n, const ClusterRules &rules,
                                   IterState *st, const QueryTrack &qt, unsigned long long *phase_log,
                                   uint32_t phase_log_iters, uint32_t leave_reads, IterState *host_st,
                                   const uint32_t *flag_src, uint32_t *flag_dst, cudaStream_t s) {
    ClusterArgs a;
    a.slots = slots;
    a.rules = rules;
    a.nm = nmats;
    a.n = n;
    a.T = (n + 63) / 64;
    a.log2r = rows_log2(n);
    a.st = st;
    a.qt = qt;
    a.phase_log = phase_log;
    a.phase_log_iters = phase_log_iters;
    a.leave_reads = leave_reads;
    a.host_st = host_st;
    a.flag_src = flag_src;
    a.flag_dst = flag_dst;
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr;
    cluster_config(&cfg, &attr, (size_t)cluster_words(a.nm, a.T, a.log2r) * 8, s);
    if (a.T <= 4) return cudaLaunchKernelEx(&cfg, k_closure_cluster<4>, a);
    if (a.T <= 8) return cudaLaunchKernelEx(&cfg, k_closure_cluster<8>, a);
    return cudaLaunchKernelEx(&cfg, k_closure_cluster<16>, a);
}

}  // namespace cfpq

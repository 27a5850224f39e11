// Variant TC: exact Boolean product C |= P * Q on the 5th-generation tensor
// cores (tcgen05.mma kind::mxf4: 4-bit operands that are non-zero where the bit
// is set, all scales 1, fp32 accumulators in TMEM, result bit = accumulator !=
// 0).  Every product is 0 or in [1/4, 4] and a sum has at most 2^17 of them, all
// of one sign: a sum is zero exactly where every product is, in any rounding.
//
// Operands travel as packed bits and are expanded on chip.  A bit keeps its
// place in a nibble: word w of the 4 words of 32 bits x is x & 0x11111111,
// x & 0x22222222, x & 0x44444444, (x >> 3) & 0x11111111 (E2M1 codes 1, 2, 4 =
// 1/2, 1, 2; code 8 would be -0).  The order of k inside 64 is then a permuted
// one, the same for both operands.
//
// 4-bit operands are K-major on both sides, so one of them has to be transposed
// bit by bit.  The block is computed as C^T = Q^T P^T: M is 128 columns of Q (2
// tiles), N is 256 rows of P (4 tiles), and it is the smaller side that is
// transposed, in registers (Transposer, 5 shuffles per 64 x 32 bits).  Work
// item (item list 2) = (product, group of 4 output tile-rows, block of 4 output
// tiles), done as two halves of 2 tile columns over the whole inner dimension.
//
// Roles (one CTA per SM, 26 warps):
//   list warp  claims items and writes the halves' k-lists (tk with an occupied
//              P tile and a non-empty Q half) into one of two list slots, an item
//              ahead: it claims when the MMAs of an item's last half start;
//   A warps    2 groups x 8: 32 columns of Q for half of a stage's k-tiles,
//              transposed and expanded to TENSOR MEMORY (tcgen05.st), from where
//              the MMA takes A;
//   B warps    2 groups x 4: one of the 4 P tiles each, expanded to shared memory
//              (no-swizzle K-major: 8-row x 16-byte core matrices);
//              group g takes the operand stages of parity g (kKt k-tiles each),
//              with the packed words loaded from global memory (L2) one unit of
//              kUnit k-tiles ahead, in the registers that the last unit left;
//   MMA warp   one tcgen05.mma (128 x 256 x 64) per k-tile, one commit per stage;
//   epilogue   the first 16 expander warps (the A warps), each after its group's
//              first stage of the next half, so that the stages fill while the
//              last MMAs drain: accumulators -> bits (64 columns a warp, transposed
//              back by shuffles) -> 4 KiB of shared memory, which frees the
//              accumulator; then one 64-bit word a lane through the atomic-OR
//              epilogue of the word-level kernels.
//
// Why this split (dense product at n = 8192, one call, 2^39 bit-MACs):
//   525 us  kind::i8, a 256 x 256 block, both operands as bytes in shared memory,
//           packed tiles by bulk copies: five copies per k-tile from one thread
//           took 1088 clocks, twice the MMAs (512);
//   408 us  128 x 256 halves with A in TMEM, words loaded straight from L2, 4
//           k-tiles per stage: a stage's 8 MMAs cost 131 clocks each where 4 per
//           commit cost 212 (one commit per about 600 clocks whatever the number
//           of stages); bound by shared memory, 128 KiB a stage at 128 B/clk;
//   262 us  4-bit operands: half the bytes through shared memory and twice the
//           MMA rate (measured 16.1 k MAC/clk per SM against 8.0 k).
// Now the integer ALU pipe bounds it: about 340 ALU instructions per k-tile (160
// for the transposed side, 80 for the plain one, 40 for the epilogue) keep it
// 70% busy and the tensor pipe 52%; the loads move 1.2 GB from L2 in that time.
//
// TMEM: accumulator 256 columns, kOpStages A stages of 8 columns a k-tile, 32
// columns of scale factors.
//
// Every wait is bounded; a wait that gives up raises the CTA's abort flag
// (which ends every other role's waits), the CTA then waits (bounded) for each
// MMA still in flight, frees TMEM and reports CFPQ_ERR_TIMEOUT.
#include <algorithm>

#include "launch.h"

namespace cfpq {

namespace {

constexpr int kAWarps = 8, kBWarps = 4;      // expanders of one stage: 128 columns of Q, 256 rows of P
constexpr int kGroupWarps = kAWarps + kBWarps;
constexpr int kBFirst = 2 * kAWarps;         // warps 0-7, 8-15: A of groups 0, 1; 16-19, 20-23: B
constexpr int kExpWarps = 2 * kGroupWarps;
constexpr int kEpiWarps = 16;                // 4 TMEM lane quarters x 4 P tiles
constexpr int kMmaWarp = kExpWarps;          // lane 0 issues the MMAs
constexpr int kListWarp = kExpWarps + 1;
constexpr int kThreads = 32 * (kExpWarps + 2);
constexpr int kMaxTiles = 2048;
constexpr unsigned kFull = 0xffffffffu;
constexpr uint32_t kN = 256;                 // output rows of an item
constexpr uint32_t kKt = 8;                  // k-tiles per operand stage: 8 MMAs per commit
constexpr uint32_t kUnit = 4;                // k-tiles whose packed words a lane holds ahead
constexpr uint32_t kOpStages = 3;            // operand stages (64 KiB and 64 TMEM columns each)
constexpr uint32_t kBTile = kN * 32;         // B operand of one k-tile
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kACol = kN, kACols = kKt * 8;         // A stages
constexpr uint32_t kSfCol = kACol + kOpStages * kACols;  // scale factors of A (16 columns) and B (16)
static_assert(kSfCol + 32 <= kTmemCols, "TMEM columns");

// Instruction descriptor, kind::mxf4: A = B = E2M1 (bits 7-9, 10-11 = 1), both
// K-major (bits 15, 16 = 0), N (bits 17-22 = N/8), scales UE8M0 (bit 23), M =
// 128 (bits 24-28 = M/16), K = 64 (bit 31 = 0).
constexpr uint32_t kIdesc = (1u << 7) | (1u << 10) | ((kN / 8) << 17) | (1u << 23) | ((128u / 16) << 24);
// B operand (K-major, no swizzle): the two 16-byte chunks of a row 128 B apart
// (LBO), 8-row groups 256 B apart (SBO).
constexpr uint32_t kBLbo = 128, kBSbo = 256;

// One item's k-lists and matrices, written by the list warp.
struct ListSlot {
    alignas(8) uint16_t ktile[2][kMaxTiles];  // padded to whole units
    uint32_t nk[2];
    uint32_t last;  // the claims ended: no item
    uint32_t ti0, tj0, T, head, query;
    const uint64_t *p, *q;
    DevMat c, d;
};

struct __align__(1024) TcSmem {
    uint8_t b[kOpStages][kKt * kBTile];  // P rows of kKt x 4 tiles
    uint32_t out[2][4][kN];              // result bits by lane quarter and row, alternate halves
    ListSlot list[2];
    uint64_t op_full[kOpStages], op_empty[kOpStages];
    uint64_t list_full[2], list_empty[2], claim;
    uint64_t acc_full, acc_empty;
    uint32_t tmem_base;
    uint32_t abort;  // a role's wait gave up: every other wait ends too
};
static_assert(sizeof(TcSmem) <= 227 * 1024, "shared memory");

__device__ __forceinline__ DevMat resolve_operand(const MatSlot &s, uint8_t use_delta, uint32_t iter) {
    if (!use_delta || iter == 0) return s.cur;
    return s.dlt[iter & 1];
}

// 64-bit shared-memory matrix descriptor, no swizzle, sm_100 version bit 46.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(sbo >> 4) << 32) |
           (1ULL << 46);
}

// D (TMEM) += A (TMEM, rows = lanes, 8 k per column) * B (shared memory)
__device__ __forceinline__ void mma_fp4(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t tmem_sf,
                                        uint32_t accumulate) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %6, 0;\n"
        " tcgen05.mma.cta_group::1.kind::mxf4.block_scale.scale_vec::2X [%0], [%1], %2, %3, [%4], [%5], p;\n}" ::"r"(
            tmem_d),
        "r"(tmem_a), "l"(bdesc), "r"(kIdesc), "r"(tmem_sf), "r"(tmem_sf + 16), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ void mma_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(bar))
                 : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// 32 lanes x 32 consecutive 32-bit TMEM columns -> 32 registers.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// 32 registers -> the lane's TMEM row, 32 columns from taddr on.
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
        "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
        "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
        "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}

// 64 bits -> 64 nibbles (8 words), non-zero where the bit is set.
__device__ __forceinline__ void expand64(uint32_t lo, uint32_t hi, uint32_t *r) {
    r[0] = lo & 0x11111111u;
    r[1] = lo & 0x22222222u;
    r[2] = lo & 0x44444444u;
    r[3] = (lo >> 3) & 0x11111111u;
    r[4] = hi & 0x11111111u;
    r[5] = hi & 0x22222222u;
    r[6] = hi & 0x44444444u;
    r[7] = (hi >> 3) & 0x11111111u;
}

// Transpose of 64 rows x 32 columns of bits, kUnit of them side by side so that
// the shuffles overlap: lane l holds rows first_row(l) and first_row(l) + 16 and
// gets column l, rows 0..31 in x[.][0] and 32..63 in x[.][1].  Step i = 4..0
// swaps the register bit of the index with bit i of the position in the word,
// then with bit i of the lane; the row bits so move through the register into the
// word, one place down each.  A lane with bit i set keeps the other register of
// the two, and the registers' order is put right by the next step's selectors.
struct Transposer {
    uint32_t keep4, send4, keep3, send3;  // byte selectors of steps 4 and 3
    uint32_t mask[3];                     // steps 0..2: bits of the lane's kept word that stay in place
    uint32_t lane;
    __device__ __forceinline__ explicit Transposer(uint32_t l) : lane(l) {
        const bool up4 = l & 16u, up3 = l & 8u;
        keep4 = up4 ? 0x7632u : 0x5410u;
        send4 = up4 ? 0x5410u : 0x7632u;
        keep3 = (up3 ? 0x7351u : 0x6240u) ^ (up4 ? 0x4444u : 0u);
        send3 = (up3 ? 0x6240u : 0x7351u) ^ (up4 ? 0x4444u : 0u);
        mask[2] = (l & 4u) ? 0xf0f0f0f0u : 0x0f0f0f0fu;
        mask[1] = (l & 2u) ? 0xccccccccu : 0x33333333u;
        mask[0] = (l & 1u) ? 0xaaaaaaaau : 0x55555555u;
    }
    static __device__ __forceinline__ uint32_t first_row(uint32_t l) { return (l >> 1) + (l & 1u) * 32; }
    __device__ __forceinline__ void operator()(uint32_t (&x)[kUnit][4]) const {
#pragma unroll
        for (uint32_t k = 0; k < kUnit; ++k) {
            const uint32_t kept = __byte_perm(x[k][0], x[k][1], keep4), sent = __byte_perm(x[k][0], x[k][1], send4);
            x[k][0] = kept;
            x[k][1] = __shfl_xor_sync(kFull, sent, 16);
        }
#pragma unroll
        for (uint32_t k = 0; k < kUnit; ++k) {
            const uint32_t kept = __byte_perm(x[k][0], x[k][1], keep3), sent = __byte_perm(x[k][0], x[k][1], send3);
            x[k][0] = kept;
            x[k][1] = __shfl_xor_sync(kFull, sent, 8);
        }
#pragma unroll
        for (int i = 2; i >= 0; --i) {
            const bool swap = ((lane >> i) ^ (lane >> (i + 1))) & 1u;
            const uint32_t s = ((lane >> i) & 1u) ? 32u - (1u << i) : 1u << i, m = mask[i];
#pragma unroll
            for (uint32_t k = 0; k < kUnit; ++k) {
                const uint32_t a = swap ? x[k][1] : x[k][0], b = swap ? x[k][0] : x[k][1];
                x[k][0] = (a & m) | (__funnelshift_l(b, b, s) & ~m);
                x[k][1] = __shfl_xor_sync(kFull, (__funnelshift_r(a, a, s) & m) | (b & ~m), 1 << i);
            }
        }
#pragma unroll
        for (uint32_t k = 0; k < kUnit; ++k) {
            const uint32_t a = x[k][0], b = x[k][1];
            x[k][0] = (lane & 1u) ? b : a;
            x[k][1] = (lane & 1u) ? a : b;
        }
    }
};

// Transpose of 32 x 32 bits: lane l holds row l and gets column l.
__device__ __forceinline__ uint32_t transpose32(uint32_t x, uint32_t lane) {
#pragma unroll
    for (int i = 4; i >= 0; --i) {
        const uint32_t s = 1u << i;
        const uint32_t m = i == 4   ? 0x0000ffffu
                           : i == 3 ? 0x00ff00ffu
                           : i == 2 ? 0x0f0f0f0fu
                           : i == 1 ? 0x33333333u
                                    : 0x55555555u;
        const uint32_t y = __shfl_xor_sync(kFull, x, s);
        x = (lane & s) ? (x & ~m) | ((y >> s) & m) : (x & m) | ((y << s) & ~m);
    }
    return x;
}

// Bounded wait that also ends when another role raised the abort flag.
__device__ __forceinline__ bool wait_or_abort(uint64_t *bar, uint32_t parity, const volatile uint32_t *abort) {
    for (uint32_t i = 0; i < kWaitLimit; ++i) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((i & 63u) == 63u && *abort) return false;
    }
    return false;
}

// A whole warp's wait: one lane giving up ends the warp's loop and the CTA.
__device__ __forceinline__ bool warp_wait(uint64_t *bar, uint32_t parity, volatile uint32_t *abort) {
    if (__all_sync(kFull, wait_or_abort(bar, parity, abort))) return true;
    *abort = 1;
    return false;
}

// The operands of one product by itself (cfpq_add_mul): the items are all
// 4 x 4-tile blocks of C in order, dealt to the CTAs by number, and the
// changed and error words go to mapped host memory -- no tables, plan or
// state.
struct TcSingle {
    DevMat a, b, c;
    const uint32_t *use_tc;  // non-null: nothing to do unless it is set
    uint32_t *host_changed, *host_error;
};

template <bool kSingle>
__global__ void __launch_bounds__(kThreads, 1)
    k_product_tc(const ProdDesc *__restrict__ prods, const MatSlot *__restrict__ slots, IterState *st,
                 const uint64_t *__restrict__ items_all, size_t list_cap, uint32_t *qchanged, BufCounters *cnts,
                 TcSingle single) {
    if (kSingle && single.use_tc && !*single.use_tc) return;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    TcSmem &S = *reinterpret_cast<TcSmem *>(smem_raw);
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    volatile uint32_t *abort = &S.abort;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&S.tmem_base)),
                     "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        for (uint32_t s = 0; s < kOpStages; ++s) {
            mbar_init(&S.op_full[s], kGroupWarps);
            mbar_init(&S.op_empty[s], 1);
        }
        for (uint32_t s = 0; s < 2; ++s) {
            mbar_init(&S.list_full[s], 1);
            mbar_init(&S.list_empty[s], kExpWarps + 1);
        }
        mbar_init(&S.claim, 1);
        mbar_init(&S.acc_full, 1);
        mbar_init(&S.acc_empty, kEpiWarps);
        S.abort = 0;
        fence_mbar_init();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = S.tmem_base;
    if (warp < 4) {  // scale factors: 1 in every byte
        uint32_t ones[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) ones[i] = 0x7f7f7f7fu;
        tmem_st32(tmem + ((32 * warp) << 16) + kSfCol, ones);
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();

    const uint32_t iter = kSingle ? 0u : st->iter;
    unsigned long long triples = 0, outw = 0, neww = 0;
    uint32_t mma_committed = 0;    // MMA warp: stages committed
    bool single_changed = false;   // (kSingle) this thread saw a new bit
    // Items, halves and operand stages are numbered through the CTA's work, by
    // every role in the same way: slot or stage = number % count, use = number /
    // count; a "full" barrier is waited with parity use & 1, an "empty" one with
    // (use & 1) ^ 1 (a fresh barrier counts its previous phase as complete, so
    // the first use passes).  A wait by parity must not come two phases early:
    // the groups take the stages by the parity of their number, not of their
    // place in the half, so that a group's wait for stage q - 2 (the MMAs of q - 5
    // are done) bounds its next one, for the MMAs of q - 3, in a row of halves
    // of one stage too.

    if (warp == kListWarp) {
        const uint64_t *const items = items_all + 2 * list_cap;
        const uint32_t blocks = (single.a.T + 3) / 4;
        const uint32_t nitems = kSingle ? blocks * blocks : st->item_count[2];
        uint32_t idx = kSingle ? blockIdx.x : 0u;
        for (uint32_t posted = 0;;) {
            // the next claim waits until the item before it is in its last half:
            // a claim far ahead would take work from CTAs that are idle
            if (posted && !warp_wait(&S.claim, (posted - 1) & 1u, abort)) break;
            if (!warp_wait(&S.list_empty[posted & 1], ((posted >> 1) & 1u) ^ 1u, abort)) break;
            ListSlot &L = S.list[posted & 1];
            uint32_t nk[2] = {0, 0};
            bool last = false;
            for (;;) {  // items until one with k-tiles
                if (!kSingle) {
                    if (lane == 0) idx = atomicAdd(&st->item_next[2], 1u);
                    idx = __shfl_sync(kFull, idx, 0);
                }
                if (idx >= nitems || *abort) {
                    last = true;
                    break;
                }
                const uint64_t it =
                    kSingle ? make_item(0, idx / blocks, idx % blocks, 0, single.a.T) : items[idx];
                if (kSingle) idx += gridDim.x;
                ProdDesc pd;
                if (kSingle) {
                    pd.T = single.a.T;
                    pd.query = 0;
                    pd.head = 0;
                } else {
                    pd = prods[item_prod(it)];
                }
                const bool merged = !kSingle && (it & kItemMerged) != 0;
                const DevMat P = kSingle ? single.a : resolve_operand(slots[pd.pslot], merged ? 0 : pd.p_delta, iter);
                const DevMat Q = kSingle ? single.b : resolve_operand(slots[pd.qslot], merged ? 0 : pd.q_delta, iter);
                const uint32_t *const dpocc = kSingle ? nullptr : slots[pd.pslot].dlt[iter & 1].occ;
                const uint32_t *const dqocc = kSingle ? nullptr : slots[pd.qslot].dlt[iter & 1].occ;
                const uint32_t T = pd.T, ow = P.ow, klo = item_klo(it), khi = item_khi(it);
                const uint32_t ti0 = item_ti(it) * 4, tj0 = item_tjb(it) * 4;
                const uint32_t qword = tj0 >> 5, qshift = tj0 & 31;
                // k-lists: tk with an occupied P tile in the 4 tile-rows and a
                // non-empty Q half, increasing tk, within the item's range; in a
                // merged item, P or Q with delta bits there
                nk[0] = nk[1] = 0;
                for (uint32_t base = 0; base < ow; base += 32) {
                    uint32_t pu = 0, du = 0;
                    if (base + lane < ow) {
                        for (uint32_t g = 0; g < min(4u, T - ti0); ++g) {
                            pu |= P.occ[(size_t)(ti0 + g) * ow + base + lane];
                            if (merged) du |= dpocc[(size_t)(ti0 + g) * ow + base + lane];
                        }
                        pu &= range_word_mask(base + lane, klo, khi);
                    }
                    for (uint32_t w0 = 0; w0 < min(32u, ow - base); w0 += 4) {
                        uint32_t mask[4];
#pragma unroll
                        for (uint32_t i = 0; i < 4; ++i) {
                            const uint32_t pw = __shfl_sync(kFull, pu, w0 + i), dw = __shfl_sync(kFull, du, w0 + i);
                            const uint32_t tk = (base + w0 + i) * 32 + lane;
                            mask[i] = 0;
                            if ((pw >> lane) & 1u)
                                mask[i] = ((!merged || ((dw >> lane) & 1u) ? Q.occ : dqocc)[(size_t)tk * ow + qword] >>
                                           qshift) & 0xFu;
                        }
#pragma unroll
                        for (uint32_t i = 0; i < 4; ++i) {
#pragma unroll
                            for (uint32_t h = 0; h < 2; ++h) {
                                const bool take = (mask[i] >> (2 * h)) & 3u;
                                const uint32_t ball = __ballot_sync(kFull, take);
                                if (take)
                                    L.ktile[h][nk[h] + __popc(ball & ((1u << lane) - 1))] =
                                        (uint16_t)((base + w0 + i) * 32 + lane);
                                nk[h] += __popc(ball);
                            }
                        }
                    }
                }
                if (!(nk[0] | nk[1])) continue;
                __syncwarp();
                if (lane < 2 * kUnit) {  // whole units: the last k-tile again
                    const uint32_t h = lane / kUnit, n = nk[h], k = (n / kUnit) * kUnit + lane % kUnit;
                    if (n && k >= n && n % kUnit) L.ktile[h][k] = L.ktile[h][n - 1];
                }
                if (lane == 0) {
                    L.nk[0] = nk[0];
                    L.nk[1] = nk[1];
                    L.ti0 = ti0;
                    L.tj0 = tj0;
                    L.T = T;
                    L.head = pd.head;
                    L.query = pd.query;
                    L.p = P.bits;
                    L.q = Q.bits;
                    L.c = kSingle ? single.c : slots[pd.head].cur;
                    if (kSingle) L.d.bits = nullptr;
                    else L.d = slots[pd.head].dlt[(iter & 1) ^ 1];
                    triples += 8ULL * (nk[0] + nk[1]);
                }
                break;
            }
            if (lane == 0) L.last = last;
            __syncwarp();
            if (lane == 0) mbar_arrive(&S.list_full[posted & 1]);
            if (last) break;
            ++posted;
        }
    } else if (warp == kMmaWarp) {
        if (lane == 0) {
            const uint64_t bdesc0 = smem_desc(smem_addr(S.b[0]), kBLbo, kBSbo);
            uint32_t seq = 0, halves = 0;
            bool ok = true;
            for (uint32_t item = 0; ok; ++item) {
                ok = wait_or_abort(&S.list_full[item & 1], (item >> 1) & 1u, abort);
                if (!ok) break;
                const ListSlot &L = S.list[item & 1];
                if (L.last) break;
                const uint32_t lasth = L.nk[1] ? 1u : 0u;
                for (uint32_t half = 0; half < 2 && ok; ++half) {
                    const uint32_t nk = L.nk[half];
                    if (half == lasth) {
                        mbar_arrive(&S.claim);
                    }
                    if (!nk) continue;
                    ok = wait_or_abort(&S.acc_empty, (halves & 1u) ^ 1u, abort);
                    if (!ok) break;
                    tc_fence_after();
                    for (uint32_t k0 = 0; k0 < nk; k0 += kKt, ++seq) {
                        const uint32_t o = seq % kOpStages;
                        ok = wait_or_abort(&S.op_full[o], (seq / kOpStages) & 1u, abort);
                        if (!ok) break;
                        tc_fence_after();
                        const uint32_t kts = min(kKt, nk - k0);
                        const uint64_t bd = bdesc0 + o * (kKt * kBTile >> 4);
#pragma unroll
                        for (uint32_t kt = 0; kt < kKt; ++kt) {
                            if (kt >= kts) break;
                            mma_fp4(tmem, tmem + kACol + o * kACols + kt * 8, bd + kt * (kBTile >> 4), tmem + kSfCol,
                                    (k0 > 0 || kt > 0) ? 1u : 0u);
                        }
                        mma_commit(&S.op_empty[o]);
                        ++mma_committed;
                    }
                    if (ok) mma_commit(&S.acc_full);  // completes after every MMA of the half
                    ++halves;
                }
                if (ok) mbar_arrive(&S.list_empty[item & 1]);
            }
            if (!ok) *abort = 1;
        }
        __syncwarp();
    } else {
        const bool is_a = warp < kBFirst;
        const uint32_t gp = is_a ? warp / kAWarps : (warp - kBFirst) / kBWarps;
        // A warp: Q tile g of the half, columns 32 hf .. of it, k-tiles kUnit sub ..
        // of a stage; B warp: P tile g, all rows and k-tiles
        const uint32_t wr = warp % 4, sub = (warp >> 2) & 1u, hf = wr & 1u;
        const uint32_t g = is_a ? wr >> 1 : wr;
        const Transposer transpose(lane);
        uint8_t *const brow = S.b[0] + (8 * g + (lane >> 3)) * kBSbo + (lane & 7) * 16;
        uint32_t seq = 0, halves = 0;
        bool pending = false;           // a half of this warp waits for its epilogue
        uint32_t pslot = 0, phalf = 0;  // its list slot and half
        bool plast = false;             // it is the item's last
        bool ok = true;
        for (uint32_t item = 0; ok; ++item) {
            ok = warp_wait(&S.list_full[item & 1], (item >> 1) & 1u, abort);
            if (!ok) break;
            ListSlot &L = S.list[item & 1];
            const bool last = L.last != 0;
            for (uint32_t half = 0; half < 2 && ok; ++half) {
                // (an end of the claims is a half without k-tiles)
                const uint32_t nk = last ? 0u : L.nk[half];
                if (!nk && !last) continue;
                const uint32_t steps = (nk + kKt - 1) / kKt, first = (gp ^ seq) & 1u;  // group gp: stages of that number parity
                const uint32_t T = L.T, tj0 = L.tj0 + 2 * half, ti0 = L.ti0;
                const uint16_t *const ktile = L.ktile[half];
                // the lane's rows of a k-tile: A first_row(lane) and 16 further of Q tile
                // g, B lane and lane + 32 of P tile g
                // (a tile beyond the matrix: its last one, whose results are not taken)
                const uint32_t tile = is_a ? min(tj0 + g, T - 1) : min(ti0 + g, T - 1);
                const char *const src = reinterpret_cast<const char *>(
                    is_a ? L.q + (size_t)tile * 64 + Transposer::first_row(lane) : L.p + tile_offset(T, tile, 0) + lane) +
                    (is_a ? 4 * hf : 0u);
                const uint32_t stride = is_a ? T * 512u : 512u;
                uint32_t ahead[kUnit][4];  // A: 32 columns of the two rows; B: both rows
                uint32_t tks[kUnit];
                const uint32_t kmax = nk ? (nk - 1) / kUnit * kUnit : 0u;
                auto ktiles = [&](uint32_t k0) {  // (lists are padded to whole units)
                    const uint2 t = *reinterpret_cast<const uint2 *>(ktile + min(k0, kmax));
                    tks[0] = t.x & 0xffffu;
                    tks[1] = t.x >> 16;
                    tks[2] = t.y & 0xffffu;
                    tks[3] = t.y >> 16;
                };
                auto load = [&](uint32_t i) {
                    const char *const at = src + (uint64_t)tks[i] * stride;
                    if (is_a) {
                        ahead[i][0] = __ldca(reinterpret_cast<const uint32_t *>(at));
                        ahead[i][1] = __ldca(reinterpret_cast<const uint32_t *>(at + 16 * 8));
                    } else {
                        const uint2 u = __ldcg(reinterpret_cast<const uint2 *>(at));
                        const uint2 v = __ldcg(reinterpret_cast<const uint2 *>(at + 32 * 8));
                        ahead[i][0] = u.x;
                        ahead[i][1] = u.y;
                        ahead[i][2] = v.x;
                        ahead[i][3] = v.y;
                    }
                };
                if (nk) {
                    ktiles(first * kKt + (is_a ? sub * kUnit : 0u));
#pragma unroll
                    for (uint32_t i = 0; i < kUnit; ++i) load(i);
                }
                for (uint32_t e = first;; e += 2) {
                    if (e < steps) {
                        const uint32_t q = seq + e, o = q % kOpStages, kts = min(kKt, nk - e * kKt);
                        ok = warp_wait(&S.op_empty[o], ((q / kOpStages) & 1u) ^ 1u, abort);
                        if (!ok) break;
                        if (is_a) {
                            tc_fence_after();
                            if (sub * kUnit < kts) {
                                uint32_t r[8 * kUnit];
                                transpose(ahead);
#pragma unroll
                                for (uint32_t i = 0; i < kUnit; ++i) expand64(ahead[i][0], ahead[i][1], r + 8 * i);
                                tmem_st32(tmem + ((32 * wr) << 16) + kACol + o * kACols + sub * kUnit * 8, r);
                                ktiles((e + 2) * kKt + sub * kUnit);
#pragma unroll
                                for (uint32_t i = 0; i < kUnit; ++i) load(i);
                                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                            }
                            tc_fence_before();
                        } else {
                            uint8_t *const at = brow + o * kKt * kBTile;
#pragma unroll
                            for (uint32_t u = 0; u < kKt; u += kUnit) {
                                if (u >= kts) break;
                                ktiles(u + kUnit < kts ? e * kKt + u + kUnit : (e + 2) * kKt);
#pragma unroll
                                for (uint32_t i = 0; i < kUnit; ++i) {
#pragma unroll
                                    for (uint32_t j = 0; j < 2; ++j) {
                                        uint32_t r[8];
                                        expand64(ahead[i][2 * j], ahead[i][2 * j + 1], r);
                                        uint8_t *const to = at + (u + i) * kBTile + 4 * j * kBSbo;
                                        *reinterpret_cast<uint4 *>(to) = make_uint4(r[0], r[1], r[2], r[3]);
                                        *reinterpret_cast<uint4 *>(to + kBLbo) = make_uint4(r[4], r[5], r[6], r[7]);
                                    }
                                    load(i);
                                }
                            }
                            fence_proxy_async_smem();  // generic-proxy writes before the tensor core reads them
                        }
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&S.op_full[o]);
                    }
                    if (pending) {
                        // ---- epilogue of the half before (number halves - 1) ----
                        pending = false;
                        const ListSlot &E = S.list[pslot];
                        const uint32_t buf = (halves - 1) & 1u, qq = warp & 3, pg = warp >> 2;
                        ok = warp_wait(&S.acc_full, buf, abort);
                        if (!ok) break;
                        tc_fence_after();
#pragma unroll
                        for (uint32_t x = 0; x < 2; ++x) {  // column of the half 32 qq + lane, rows 64 pg + 32 x ..
                            uint32_t v[32];
                            tmem_ld32(tmem + ((32 * qq) << 16) + pg * 64 + x * 32, v);
                            uint32_t w = 0;
#pragma unroll
                            for (int c = 0; c < 32; ++c) w = __funnelshift_l(__float_as_uint(0.0f - __uint_as_float(v[31 - c])), w, 1);
                            S.out[buf][qq][pg * 64 + x * 32 + lane] = transpose32(w, lane);
                        }
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&S.acc_empty);  // the accumulator may be overwritten
                        ok = warp_wait(&S.acc_empty, buf, abort);  // every warp's bits are there
                        if (!ok) break;
                        const uint32_t jt = (warp >> 1) & 1u, r = (warp & 1u) * 32 + lane;
                        const uint32_t ti = E.ti0 + pg, tj = E.tj0 + 2 * phalf + jt;
                        const uint64_t a = (uint64_t)S.out[buf][2 * jt][pg * 64 + r] |
                                           ((uint64_t)S.out[buf][2 * jt + 1][pg * 64 + r] << 32);
                        uint32_t newcnt = 0;
                        if (a && ti < E.T && tj < E.T) {
                            ++outw;
                            const size_t off = tile_offset(E.T, ti, tj) + r;
                            unsigned long long *cw = reinterpret_cast<unsigned long long *>(E.c.bits + off);
                            const uint64_t seen = __ldcg(cw);
                            if (a & ~seen) {
                                const uint64_t prev = atomicOr(cw, (unsigned long long)a);
                                const uint64_t nw = a & ~prev;
                                if (nw) {
                                    ++neww;
                                    newcnt = __popcll(nw);
                                    if (E.d.bits)
                                        atomicOr(reinterpret_cast<unsigned long long *>(E.d.bits + off),
                                                 (unsigned long long)nw);
                                }
                            }
                        }
                        const uint32_t tile_new = __reduce_add_sync(kFull, newcnt);  // 32 rows of one tile
                        if (tile_new) {  // lane 0: tile tj (populations, occupancy, counters)
                            const uint32_t mine = lane == 0 ? tile_new : 0u;
                            tiles_gain(E.c, ti, tj, mine, cnts ? cnts + 3 * E.head : nullptr);
                            if (E.d.bits)
                                tiles_gain(E.d, ti, tj, mine, cnts ? cnts + 3 * E.head + 1 + ((iter & 1) ^ 1) : nullptr);
                            if (kSingle) {
                                single_changed = true;
                            } else if (lane == 0) {
                                st->changed = 1u;
                                if (qchanged) qchanged[E.query] = 1u;
                            }
                        }
                        __syncwarp();
                        if (plast && lane == 0) mbar_arrive(&S.list_empty[pslot]);
                    }
                    if (e + 2 >= steps) break;
                }
                if (!nk || !ok) break;
                seq += steps;
                ++halves;
                const bool final_half = half == 1 || !L.nk[1];
                if (warp < kEpiWarps) {
                    pending = true;
                    pslot = item & 1;
                    phalf = half;
                    plast = final_half;
                } else if (final_half) {
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&S.list_empty[item & 1]);
                }
                if (final_half) break;  // the slot may already hold another item
            }
            if (last) break;
        }
    }

    // ---- exit: after a wait gave up, wait (bounded) for every MMA still in
    // flight before TMEM is freed and the CTA ends ----
    __syncthreads();
    const bool aborted = *abort != 0;
    if (aborted && warp == kMmaWarp && lane == 0 && mma_committed) {
        // the last commit completes after every MMA issued before it
        const uint32_t q = mma_committed - 1;
        mbar_wait_bounded(&S.op_empty[q % kOpStages], (q / kOpStages) & 1u);
    }
    if (kSingle) {
        const bool changed = __syncthreads_or(single_changed) != 0;
        if (changed && tid == 0) *single.host_changed = 1u;
        if (aborted && tid == 0) *single.host_error = 5u;
    } else {
        for (int o = 16; o > 0; o >>= 1) {
            triples += __shfl_down_sync(kFull, triples, o);
            outw += __shfl_down_sync(kFull, outw, o);
            neww += __shfl_down_sync(kFull, neww, o);
        }
        if (lane == 0) {
            if (triples) atomicAdd(&st->tile_triples, triples);
            if (outw) atomicAdd(&st->out_words, outw);
            if (neww) atomicAdd(&st->new_words, neww);
        }
        if (aborted && tid == 0) atomicExch(&st->error, 5u);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
}

}  // namespace

int product_tc_blocks_per_sm() {
    cudaFuncSetAttribute(k_product_tc<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(TcSmem));
    cudaFuncSetAttribute(k_product_tc<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(TcSmem));
    int nb = 0, nb1 = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_product_tc<false>, kThreads, sizeof(TcSmem));
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb1, k_product_tc<true>, kThreads, sizeof(TcSmem));
    return nb == nb1 ? nb : 0;
}

cudaError_t launch_product_tc(const ProdDesc *d_prods, const MatSlot *d_slots, IterState *d_st,
                              const uint64_t *d_items, size_t list_cap, uint32_t *d_qchanged, int grid,
                              BufCounters *cnts, cudaStream_t s) {
    k_product_tc<false><<<grid, kThreads, sizeof(TcSmem), s>>>(d_prods, d_slots, d_st, d_items, list_cap, d_qchanged,
                                                               cnts, TcSingle{});
    return cudaGetLastError();
}

cudaError_t launch_add_mul_tc(const DevMat &a, const DevMat &b, const DevMat &c, int grid, const uint32_t *use_tc,
                              uint32_t *host_changed, uint32_t *host_error, cudaStream_t s) {
    if (a.T == 0) return cudaSuccess;
    const uint32_t blocks = (a.T + 3) / 4;
    k_product_tc<true><<<std::min((uint32_t)grid, blocks * blocks), kThreads, sizeof(TcSmem), s>>>(
        nullptr, nullptr, nullptr, nullptr, 0, nullptr, nullptr, TcSingle{a, b, c, use_tc, host_changed, host_error});
    return cudaGetLastError();
}

}  // namespace cfpq

// Paged prefill attention on the 5th-generation tensor cores (tcgen05), bfloat16,
// head sizes 64 and 128, page sizes that are powers of two from 8.
//
// Work unit: 128 query rows x one kv head; the rows of a request are flattened as
// rho = local_token * g + head_in_group (whole tokens per tile: floor(128 / g) of
// them), so the g query heads of a group share every key/value tile.  Per 64-key
// tile, with both accumulators in tensor memory (TMEM):
//
//   loader warps    TMA tensor copies (128-byte swizzle) of the queries, then of the tile's pages of K (warp 0)
//                   and of V (warp 6) into two-stage shared-memory rings of their own
//                                                          -> k_full[stage], v_full[stage]
//   MMA warp        S = Q.K^T   (tcgen05.mma M=128 N=64,  K=16 x D/16)  -> s_full (scores ready,
//                                                                          keys may be replaced)
//                   O += P.V    (tcgen05.mma M=128 N=D,   K=16 x 4)     -> pv_done (values may
//                                                                          be replaced, O is final)
//   softmax warps   thread r owns row r: tcgen05.ld its 64 scores, mask, running max and
//                   sum in float32 (no shuffles: a row lives in one thread), P as
//                   bfloat16 back into tensor memory (tcgen05.st, over the scores it
//                   came from), where the second MMA reads its A operand  -> p_full
// The scores are double buffered: Q.K^T of the next tile runs while this tile's softmax
// does, and P of a tile never waits for the P.V of the one before.  Every barrier that
// is waited on by parity is one of a pair indexed by the tile's buffer, so that the
// side that signals can never be two phases ahead of the side that waits: the softmax
// warps may finish tile j + 1 before the MMA warp has seen P of tile j (both score
// buffers are filled ahead), and a single "P is ready" barrier would then have wrapped
// past the phase the MMA warp still waits for.
//
// The running maximum is only raised when the tile's maximum exceeds it by more than
// 2^8 (scores are in the base-2 domain); otherwise the stale maximum keeps being used
// (probabilities stay below 256, exact in the float32 sums), so the accumulator in
// TMEM is rescaled rarely.  Two blocks fit on an SM: one does its softmax while the
// other's MMAs run.
//
// What bounds it: a tile's 64 exponentials a row (512 cycles a block and tile, 700 reached with two blocks an
// SM) and about 4 us of look-ups, first copies and result a block.  The queries come by one copy a panel, and only
// rows that no copy brings are zeroed, by the loaders.  A few long tiles (a portion of a prompt late in its request)
// leave SMs empty: then the blocks of a cluster share a tile's keys and add their parts up through shared memory
// (`splits`).  us before these and the packed arithmetic -> now: 2,048 tokens of 28 / 4 heads of 128 43.5 -> 39.3, 14 / 2
// heads of 64 30.2 -> 26.4; 449 tokens after 512 beside 31 single ones, 14 / 2 heads 17.3 -> 14.8; 16 tokens after
// 1,500 22.4 -> 10.6.
//
// Every mbarrier wait is bounded; a role that gives up records a code in the status
// word and leaves its loop; the block then frees its TMEM and returns without a result, and so do the blocks that
// share keys with it.
//
// Reference analogue: the torch loop over sequences (servelab/parallel/
// tp_model.py:136-157); masking and softmax follow it (r <= a, optional window).
#include <cuda.h>

#include "softmax_util.cuh"
#include "tma_util.cuh"

#if (SLB_HEAD_DIM == 64 || SLB_HEAD_DIM == 128)

namespace {

constexpr int D = SLB_HEAD_DIM;
constexpr int PANELS = D / 64;                 // 64-element (128-byte) column panels
constexpr int BM = 128, BN = 64;
constexpr int THREADS = 224;                   // warp 0 loads keys, 1 issues the MMAs, 2..5 softmax,
                                               // 6 loads values
constexpr int TMEM_COLS = 256;                 // two S buffers at columns 0..127, O at 128..128+D-1
constexpr int S_COL = 0, O_COL = 128;          // S buffer b sits at S_COL + 64 * b
constexpr int Q_BYTES = PANELS * BM * 128;
constexpr int KV_PANEL_BYTES = BN * 128;
constexpr int KV_TILE_BYTES = PANELS * KV_PANEL_BYTES;
constexpr int OFF_Q = 0;
constexpr int OFF_K = OFF_Q + Q_BYTES;
constexpr int OFF_V = OFF_K + 2 * KV_TILE_BYTES;
constexpr int OFF_BAR = OFF_V + 2 * KV_TILE_BYTES;
constexpr int OFF_ML = OFF_BAR + 128;          // a row's reference and sum, for the blocks that share its keys
constexpr int OFF_GAVE = OFF_ML + BM * 8;      // ... and whether this block gave up
constexpr size_t TC_ATTN_SMEM = OFF_GAVE + 16;
constexpr int MAX_SPLITS = 8;
static_assert(OFF_BAR - OFF_K >= BM * D * 4, "the rings hold a block's partial result");
constexpr uint32_t SPIN_LIMIT = 1u << 18;     // a poll that suspends takes about 4 us: about a second
constexpr float RESCALE_THRESHOLD = 8.f;       // log2 of the largest probability tolerated

__device__ int tc_attn_status = 0;
// Where bounded waits gave up last, four ints per role (loader, MMA issuer, softmax):
// code, block, key tile, key tiles of the block.
__device__ int tc_attn_where[12] = {0};

__device__ __forceinline__ void gave_up(int* status, int code, int role, int tile, int ntiles) {
    atomicCAS(status, 0, code);
    tc_attn_where[role * 4 + 0] = code;
    tc_attn_where[role * 4 + 1] = (int)blockIdx.x;
    tc_attn_where[role * 4 + 2] = tile;
    tc_attn_where[role * 4 + 3] = ntiles;
}

using slb_tma::tma_load_2d;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}
// Bounded wait for the phase of the given parity, entered by a whole warp: false in every lane if it ran out in one.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
    const uint32_t addr = smem_u32(bar);
    uint32_t done = 0;
    for (uint32_t i = 0; i < SPIN_LIMIT && !done; ++i)
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done) : "r"(addr), "r"(parity) : "memory");
    return slb_warp_agrees(done != 0);
}
// The same wait for hand-overs on the critical path of a tile (scores ready, P ready):
// test_wait does not suspend the thread, so the waiter sees the phase within tens of
// cycles; bounded by SPIN_LIMIT * 64 polls (a poll that does not suspend is ~60 times
// shorter).
__device__ __forceinline__ bool mbar_spin(uint64_t* bar, uint32_t parity) {
    const uint32_t addr = smem_u32(bar);
    uint32_t done = 0;
    for (uint32_t i = 0; i < SPIN_LIMIT * 64u && !done; ++i)
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done) : "r"(addr), "r"(parity) : "memory");
    return slb_warp_agrees(done != 0);
}
// Shared-memory matrix descriptor, 128-byte swizzle, rows of 128 bytes in groups of 8
// (1024 bytes).  lbo16: leading byte offset >> 4 (distance of 64-element panels for an
// operand that is contiguous along M/N; unused for K-major operands).
__device__ __forceinline__ uint64_t umma_desc(uint32_t smem_addr, uint32_t lbo16) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr >> 4) & 0x3FFF);
    d |= (uint64_t)(lbo16 & 0x3FFF) << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}
__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                          uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// same with the A operand in tensor memory (lane = row, 32-bit columns of two bfloat16)
__device__ __forceinline__ void umma_bf16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc,
                                             uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                 ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
          "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
          "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
          "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr));
}
// the 64 scores of this thread's row
__device__ __forceinline__ void tmem_ld64(uint32_t taddr, float (&s)[64]) {
    uint32_t v[2][32];
    tmem_ld32(taddr, v[0]);
    tmem_ld32(taddr + 32, v[1]);
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 64; ++i) s[i] = __uint_as_float(v[i >> 5][i & 31]);
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
        "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
        ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
          "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]),
          "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]),
          "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
        : "memory");
}
using slb_softmax::pack2;
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// the float at `mine` in block `rank` of the cluster
__device__ __forceinline__ float cluster_float(const float* mine, uint32_t rank) {
    uint32_t a;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(mine)), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
    return v;
}

__global__ void __launch_bounds__(THREADS, 2) prefill_attention_tc_kernel(
    const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
    const __grid_constant__ CUtensorMap map_v, bf16* __restrict__ out, int ldo,
    const int* __restrict__ block_table, int max_pages, const int* __restrict__ cu_q,
    const int* __restrict__ ctx_len, const int* __restrict__ tile_seq, const int* __restrict__ tile_row0,
    int H, int Hkv, int ps, int box_rows, float scale_log2, int window, int splits, int* __restrict__ status) {
    extern __shared__ __align__(1024) unsigned char smem[];
    // All barriers come in pairs indexed by tile parity.  s_full[b]: Q.K^T of a tile is done
    // (its scores are ready and its keys may be replaced); pv_done[b]: its P.V is done (its
    // values may be replaced, the accumulator may be rescaled or read).
    uint64_t* k_full = reinterpret_cast<uint64_t*>(smem + OFF_BAR);     // [2]
    uint64_t* v_full = k_full + 2;                                      // [2]
    uint64_t* s_full = v_full + 2;                                      // [2]
    uint64_t* p_full = s_full + 2;                                      // [2], one per score buffer
    uint64_t* pv_done = p_full + 2;                                     // [2]
    uint64_t* q_full = pv_done + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(q_full + 1);

    pdl_wait();
    const int warp = slb_warp(), lane = threadIdx.x & 31;
    // Blocks are handed out in the order of their linear index: tile by tile from the last
    // (most keys) to the first, all kv heads of a tile together, so that no head's long
    // tiles start late.
    const int rank = (int)blockIdx.x % splits, unit = (int)blockIdx.x / splits, units = (int)gridDim.x / splits;
    const int kvh = unit % Hkv;
    const int tile = units / Hkv - 1 - unit / Hkv;
    const int s = tile_seq[tile];
    const int row0 = tile_row0[tile];
    const int g = H / Hkv;
    const int q0 = cu_q[s];
    const int qlen = cu_q[s + 1] - q0;
    const int ctx = ctx_len[s];
    const int rows_per_tile = (BM / g) * g;
    const int nrows = min(rows_per_tile, qlen * g - row0);
    const int tok0 = row0 / g;
    const int pos_base = ctx - qlen;
    const int* table = block_table + (size_t)s * max_pages;
    const bool aligned = (smem_u32(smem) & 1023u) == 0;     // the swizzle needs 1024-byte alignment
    if (nrows <= 0 || !aligned) {                            // (every block of a cluster, or none)
        if (!aligned && threadIdx.x == 0) atomicCAS(status, 0, 0x900);
        return;
    }
    const int p_first = pos_base + tok0;
    const int p_last = pos_base + tok0 + (nrows - 1) / g;
    int kbeg = 0;
    if (window > 0) kbeg = max(0, p_first - window + 1) / BN * BN;
    int kend = p_last + 1;
    int ntiles = (kend - kbeg + BN - 1) / BN;
    if (splits > 1) {                                       // this block's share of the keys (maybe none)
        const int per = (ntiles + splits - 1) / splits, first = min(ntiles, rank * per);
        ntiles = min(ntiles, first + per) - first;
        kbeg += first * BN;
        kend = min(kend, kbeg + ntiles * BN);
    }

    if (threadIdx.x == 0) {
        for (int i = 0; i < 2; ++i) {
            mbar_init(&k_full[i], 1);
            mbar_init(&v_full[i], 1);
            mbar_init(&pv_done[i], 1);
        }
        mbar_init(q_full, 1);
        *reinterpret_cast<volatile int*>(smem + OFF_GAVE) = 0;
        mbar_init(&s_full[0], 1); mbar_init(&s_full[1], 1);
        mbar_init(&p_full[0], 128); mbar_init(&p_full[1], 128);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(tmem_slot)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;

    if (warp == 0 || warp == 6) {
        // ---------------------------------------------------------------- loaders
        // Warp 0 fetches the keys, warp 6 the values, each through its own two-stage ring:
        // the keys of a tile may be replaced when its Q.K^T has run (two softmax periods
        // before the new ones are needed), the values when its P.V has.  Lane b looks up the
        // page of box b, one tile ahead of its use (a dependent global load).
        const bool keys = warp == 0;
        const CUtensorMap* map = keys ? &map_k : &map_v;
        unsigned char* ring = smem + (keys ? OFF_K : OFF_V);
        uint64_t* full = keys ? k_full : v_full;
        uint64_t* freed = keys ? s_full : pv_done;
        const int boxes = BN / box_rows;
        const int shift = __ffs(ps) - 1;                  // the launcher only takes powers of two
        auto lookup = [&](int j) {                        // first cache row of this lane's box, or -1
            int row = -1;
            if (lane < boxes && j < ntiles) {
                const int kp = kbeg + j * BN + lane * box_rows;
                if (kp < kend) {
                    const int page = table[kp >> shift];
                    if (page >= 0) row = (page * Hkv + kvh) * ps + (kp & (ps - 1));
                }
            }
            return row;
        };
        if (keys && ntiles > 0 && slb_elected()) {          // the queries: whole tokens, a panel a copy (rows beyond the
            mbar_expect_tx(q_full, PANELS * (BM / g) * g * 128);               // tile's are computed and not stored)
#pragma unroll
            for (int p = 0; p < PANELS; ++p)
                slb_tma::tma_load_3d(smem + OFF_Q + p * (BM * 128), &map_q, q_full, p * 64, kvh * g, q0 + tok0);
        }
        int row = lookup(0), asked = 0;
        for (int j = 0; j < ntiles; ++j, ++asked) {
            const int st = j & 1;
            const int next_row = lookup(j + 1);
            if (!mbar_wait(&freed[st], ((j >> 1) & 1) ^ 1)) {
                if (lane == 0) gave_up(status, keys ? 0x101 : 0x102, 0, j, ntiles);
                break;
            }
            const unsigned got = __ballot_sync(0xffffffffu, row >= 0);
            if (got != (1u << boxes) - 1u) {               // rows that no copy brings (absent pages) hold zeros
                for (int b = 0; b < boxes; ++b) {
                    if (got >> b & 1u) continue;
                    slb_tma::zero_box(ring + st * KV_TILE_BYTES + b * box_rows * 128, PANELS, KV_PANEL_BYTES, box_rows * 128,
                                      lane);
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
            }
            if (slb_elected()) {
                const uint32_t bytes = (uint32_t)__popc(got) * (uint32_t)box_rows * 128u * PANELS;
                if (bytes) mbar_expect_tx(&full[st], bytes); else mbar_arrive(&full[st]);
            }
            for (int b = 0; b < boxes; ++b) {
                const int box_row = __shfl_sync(0xffffffffu, row, b);
                if (box_row >= 0 && slb_elected()) {
#pragma unroll
                    for (int p = 0; p < PANELS; ++p)
                        tma_load_2d(ring + st * KV_TILE_BYTES + p * KV_PANEL_BYTES + b * box_rows * 128, map, &full[st],
                                    p * 64, box_row);
                }
            }
            row = next_row;
        }
        // (after a wait that gave up copies may be in flight, which must not land in a later block's memory: the last of each
        // stage is waited for; otherwise the MMAs have waited for them)
        for (int t = max(0, asked - 2); t < asked; ++t) mbar_wait(&full[t & 1], (t >> 1) & 1);
        if (keys && ntiles > 0) mbar_wait(q_full, 0);
    } else if (warp == 1) {
        // ---------------------------------------------------------------- MMA issuer
        const uint32_t idesc_qk = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) |
                                  ((uint32_t)(BM >> 4) << 24);
        const uint32_t idesc_pv = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) |
                                  ((uint32_t)(D >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
        // operand descriptors are built once; a step along K or to another panel adds its
        // byte offset / 16 to the address field
        const uint64_t q_desc = umma_desc(smem_u32(smem + OFF_Q), 1);
        const uint64_t k_desc0 = umma_desc(smem_u32(smem + OFF_K), 1);
        const uint64_t v_desc0 = umma_desc(smem_u32(smem + OFF_V), KV_PANEL_BYTES >> 4);
        constexpr uint64_t STAGE_STEP = KV_TILE_BYTES >> 4;      // to the second stage
        // S = Q.K^T of tile t into score buffer t & 1 (which held the scores and then P of
        // tile t - 2; its P.V has been issued before)
        auto issue_qk = [&](int t) -> bool {
            const int st = t & 1;
            if (!mbar_spin(&k_full[st], (t >> 1) & 1)) { gave_up(status, 0x201, 1, t, ntiles); return false; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (slb_elected()) {
#pragma unroll
                for (int p = 0; p < PANELS; ++p)
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk)          // 16 elements of D = 32 bytes per step
                        umma_bf16(tmem + S_COL + 64 * st, q_desc + ((p * (BM * 128) + kk * 32) >> 4),
                                  k_desc0 + st * STAGE_STEP + ((p * KV_PANEL_BYTES + kk * 32) >> 4), idesc_qk,
                                  (p > 0 || kk > 0) ? 1u : 0u);
                umma_commit(&s_full[st]);
            }
            return true;
        };
        bool ok = true;
        if (ntiles > 0 && !mbar_spin(q_full, 0)) { gave_up(status, 0x204, 1, 0, ntiles); ok = false; }
        if (ok && ntiles > 0) ok = issue_qk(0);
        if (ok && ntiles > 1) ok = issue_qk(1);
        for (int j = 0; j < ntiles && ok; ++j) {
            const int st = j & 1;
            if (!mbar_spin(&p_full[st], (j >> 1) & 1)) { gave_up(status, 0x202, 1, j, ntiles); break; }
            if (!mbar_spin(&v_full[st], (j >> 1) & 1)) { gave_up(status, 0x203, 1, j, ntiles); break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (slb_elected()) {
#pragma unroll
                for (int kk = 0; kk < 4; ++kk)              // 16 keys per step: P 8 columns, V 16 rows
                    umma_bf16_ts(tmem + O_COL, tmem + S_COL + 64 * st + kk * 8,
                                 v_desc0 + st * STAGE_STEP + ((kk * 16 * 128) >> 4), idesc_pv,
                                 (j > 0 || kk > 0) ? 1u : 0u);
                umma_commit(&pv_done[st]);
            }
            // the scores of tile j + 2 go where P of tile j was: issued after P.V of tile j
            // (the tensor core executes in issue order), while the softmax of j + 1 runs
            if (j + 2 < ntiles) ok = issue_qk(j + 2);
        }
    } else {
        // ---------------------------------------------------------------- softmax + epilogue
        const int quarter = warp & 3;
        const int r = quarter * 32 + lane;
        const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
        const int pos = r < nrows ? pos_base + tok0 + r / g : -1;
        float m_ref = -INFINITY, l = 0.f;
        bool ok = true;
        const bool live = quarter * 32 < nrows;             // (a warp whose rows are all padding only hands tiles on)
        for (int j = 0; j < ntiles && ok; ++j) {
            if (!(live ? mbar_spin(&s_full[j & 1], (j >> 1) & 1) : mbar_wait(&s_full[j & 1], (j >> 1) & 1))) {
                if (lane == 0) gave_up(status, 0x301, 2, j, ntiles);
                ok = false;
                break;
            }
            if (!live) {
                mbar_arrive(&p_full[j & 1]);
                continue;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            float s[64];
            tmem_ld64(tmem + lane_base + S_COL + 64 * (j & 1), s);
            const int k0 = kbeg + j * BN;
            // raw scores stay unscaled; masked ones become -inf.  A tile that every row of
            // the block sees completely needs no mask (rows of padding compute garbage that
            // is never stored).
            const bool open = k0 + BN - 1 <= p_first && k0 + BN <= kend && (window <= 0 || p_last - k0 < window);
            if (!open) slb_softmax::mask_keys(s, window > 0 ? pos - window + 1 - k0 : 0, min(kend, pos + 1) - k0);
            const float mt = slb_softmax::max_of(s) * scale_log2;     // scale > 0
            float alpha = 1.f;
            if (mt > m_ref + RESCALE_THRESHOLD || (m_ref == -INFINITY && mt != -INFINITY)) {
                alpha = (m_ref == -INFINITY) ? 0.f : exp2f(m_ref - mt);
                m_ref = mt;
            }
            uint32_t packed[32];
            l = l * alpha + slb_softmax::exponentials(s, scale_log2, m_ref == -INFINITY ? 0.f : m_ref, packed);
            if (j > 0 && __any_sync(0xffffffffu, alpha != 1.f)) {
                // the accumulator is rescaled (rarely): P.V of the previous tile must be done
                if (!mbar_wait(&pv_done[(j - 1) & 1], ((j - 1) >> 1) & 1)) { if (lane == 0) gave_up(status, 0x302, 2, j, ntiles); ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                for (int c0 = 0; c0 < D; c0 += 32) {
                    uint32_t ov[32];
                    tmem_ld32(tmem + lane_base + O_COL + c0, ov);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int i = 0; i < 32; ++i) ov[i] = __float_as_uint(__uint_as_float(ov[i]) * alpha);
                    tmem_st32(tmem + lane_base + O_COL + c0, ov);
                }
            }
            // P: 64 bfloat16 = 32 columns, written over the first half of this tile's scores
            tmem_st32(tmem + lane_base + S_COL + 64 * (j & 1), packed);
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            mbar_arrive(&p_full[j & 1]);
        }
        if (ok && ntiles > 0) {
            if (!mbar_wait(&pv_done[(ntiles - 1) & 1], ((ntiles - 1) >> 1) & 1)) { if (lane == 0) gave_up(status, 0x303, 2, ntiles, ntiles); ok = false; }
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        pdl_launch_dependents();
        if (splits == 1) {
            const float inv = l > 0.f ? 1.f / l : 0.f;
            const int tl = r / g, hg = r - tl * g;
            bf16* dst = out + (size_t)(q0 + tok0 + tl) * ldo + (size_t)(kvh * g + hg) * D;
#pragma unroll
            for (int c0 = 0; c0 < D; c0 += 32) {
                uint32_t ov[32];
                tmem_ld32(tmem + lane_base + O_COL + c0, ov);        // warp-wide: every lane takes part
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (ok && r < nrows) {
#pragma unroll
                    for (int i = 0; i < 32; i += 8) {
                        uint4 v;
                        v.x = pack2(__uint_as_float(ov[i]) * inv, __uint_as_float(ov[i + 1]) * inv);
                        v.y = pack2(__uint_as_float(ov[i + 2]) * inv, __uint_as_float(ov[i + 3]) * inv);
                        v.z = pack2(__uint_as_float(ov[i + 4]) * inv, __uint_as_float(ov[i + 5]) * inv);
                        v.w = pack2(__uint_as_float(ov[i + 6]) * inv, __uint_as_float(ov[i + 7]) * inv);
                        *reinterpret_cast<uint4*>(dst + c0 + i) = v;
                    }
                }
            }
        } else {
            // This block's part of the result, for the other blocks of the row: columns of a thread's row side by side in the
            // idle rings, and (reference, sum); a block without keys counts for nothing, after one that gave up no block
            // of the cluster has a result.
            float* part = reinterpret_cast<float*>(smem + OFF_K);
            float* ml = reinterpret_cast<float*>(smem + OFF_ML);
            const bool counts = ok && ntiles > 0;
            if (!ok) *reinterpret_cast<volatile int*>(smem + OFF_GAVE) = 1;
            ml[r * 2] = counts ? m_ref : -INFINITY;
            ml[r * 2 + 1] = counts ? l : 0.f;
            if (ntiles > 0) {
#pragma unroll
                for (int c0 = 0; c0 < D; c0 += 32) {
                    uint32_t ov[32];
                    tmem_ld32(tmem + lane_base + O_COL + c0, ov);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int i = 0; i < 32; ++i) part[(c0 + i) * BM + r] = counts ? __uint_as_float(ov[i]) : 0.f;
                }
            }
        }
    }
    if (splits > 1) {
        __syncwarp();
        cluster_sync();
        if (warp >= 2 && warp < 6) {
            // Thread r finishes its row's share of the columns, the blocks' parts added in their order.
            const int r = (warp & 3) * 32 + lane, tl = r / g, hg = r - tl * g;
            const float* part = reinterpret_cast<const float*>(smem + OFF_K);
            const float* ml = reinterpret_cast<const float*>(smem + OFF_ML);
            float m = -INFINITY, l = 0.f, w[MAX_SPLITS];
            bool whole = true;                               // (no block's part is missing)
            for (int k = 0; k < splits; ++k) {
                m = fmaxf(m, cluster_float(ml + r * 2, k));
                whole = whole && __float_as_int(cluster_float(reinterpret_cast<const float*>(smem + OFF_GAVE), k)) == 0;
            }
#pragma unroll
            for (int k = 0; k < MAX_SPLITS; ++k) {
                w[k] = 0.f;
                if (k >= splits) continue;
                const float mk = cluster_float(ml + r * 2, k);
                if (mk != -INFINITY) w[k] = exp2f(mk - m);
                l += w[k] * cluster_float(ml + r * 2 + 1, k);
            }
            const float inv = l > 0.f ? 1.f / l : 0.f;
            const int share = D / splits;                    // (a multiple of 8)
            bf16* dst = out + (size_t)(q0 + tok0 + tl) * ldo + (size_t)(kvh * g + hg) * D;
            if (whole && r < nrows) {
                for (int c = rank * share; c < (rank + 1) * share; c += 8) {
                    float o[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
                    for (int k = 0; k < MAX_SPLITS; ++k) {
                        if (k >= splits || w[k] == 0.f) continue;
#pragma unroll
                        for (int i = 0; i < 8; ++i) o[i] += w[k] * cluster_float(part + (c + i) * BM + r, k);
                    }
                    uint4 v;
                    v.x = pack2(o[0] * inv, o[1] * inv); v.y = pack2(o[2] * inv, o[3] * inv);
                    v.z = pack2(o[4] * inv, o[5] * inv); v.w = pack2(o[6] * inv, o[7] * inv);
                    *reinterpret_cast<uint4*>(dst + c) = v;
                }
            }
        }
        __syncwarp();
        cluster_sync();                                      // (the parts stay until every block has read them)
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS)
                     : "memory");
    }
}

// the cache of one layer as a matrix [pages * kv heads * page size, D]; boxes of box_rows x 64
int make_cache_map(CUtensorMap* map, const void* ptr, long long rows, int box_rows) {
    return slb_tma::make_rows_map(map, ptr, D, rows, box_rows);
}

}  // namespace

extern "C" {

// 1 if the (head size, page size, group size) is taken by the tcgen05 prefill kernel
int slb_prefill_attention_tc_supported(int ps, int group) {
    return ps >= 8 && (ps & (ps - 1)) == 0 && group >= 1 && group <= BM;
}
// query rows per tile for a group of g query heads (whole tokens per tile)
int slb_prefill_attention_tc_tile_rows(int group) { return group >= 1 && group <= BM ? (BM / group) * group : 0; }

// num_pages: pages in k_cache / v_cache ([num_pages][Hkv][ps][D]).
// tokens: rows of q.  splits: blocks (a cluster) that share the keys of a tile of rows, 1, 2, 4 or 8.
int slb_prefill_attention_tc_bf16(const bf16* q, int ldq, int tokens, const bf16* kc, const bf16* vc, bf16* out, int ldo,
                                  const int* block_table, int max_pages, const int* cu_q,
                                  const int* ctx_len, const int* tile_seq, const int* tile_row0,
                                  int num_tiles, int H, int Hkv, int ps, int num_pages, float scale,
                                  int window, int splits, cudaStream_t st) {
    if (num_tiles <= 0) return 0;
    if (tokens <= 0 || (splits != 1 && splits != 2 && splits != 4 && splits != 8)) return SLB_ERR_BAD_ARG;
    if (H <= 0 || Hkv <= 0 || H % Hkv != 0 || max_pages <= 0 || num_pages <= 0 || !(scale > 0.f))
        return SLB_ERR_BAD_ARG;
    if (!slb_prefill_attention_tc_supported(ps, H / Hkv)) return SLB_ERR_BAD_ARG;
    if (ldq % 8 || ldo % 8 || ((uintptr_t)q | (uintptr_t)kc | (uintptr_t)vc | (uintptr_t)out) % 16)
        return SLB_ERR_BAD_ARG;
    if ((long long)num_tiles * Hkv * splits > 0x7fffffffll) return SLB_ERR_TOO_LARGE;
    const int box_rows = ps < BN ? ps : BN;
    CUtensorMap map_q, map_k, map_v;
    const int g = H / Hkv;
    const long long rows = (long long)num_pages * Hkv * ps;
    if (rows > 0x7fffffffll) return SLB_ERR_TOO_LARGE;    // box coordinates are 32-bit
    // (a block-table entry outside [0, num_pages) names rows outside the tensor map: the copy
    // reads zeros there, never memory outside the cache)
    int rc = slb_tma::make_query_map(&map_q, q, D, H, tokens, ldq, g, BM / g);
    if (rc != 0) return rc;
    rc = make_cache_map(&map_k, kc, rows, box_rows);
    if (rc != 0) return rc;
    rc = make_cache_map(&map_v, vc, rows, box_rows);
    if (rc != 0) return rc;
    static unsigned long long configured = 0;              // a bit per device
    rc = slb_configure(&configured, prefill_attention_tc_kernel, TC_ATTN_SMEM);
    if (rc != 0) return rc;
    int* status = nullptr;
    cudaError_t e = cudaGetSymbolAddress((void**)&status, tc_attn_status);
    if (e != cudaSuccess) return (int)e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)num_tiles * Hkv * splits);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = TC_ATTN_SMEM;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)splits;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = slb_pdl_enabled ? attr : attr + 1;
    cfg.numAttrs = (slb_pdl_enabled ? 1 : 0) + (splits > 1 ? 1 : 0);
    return (int)cudaLaunchKernelEx(&cfg, prefill_attention_tc_kernel, map_q, map_k, map_v, out, ldo, block_table, max_pages,
                                   cu_q, ctx_len, tile_seq, tile_row0, H, Hkv, ps, box_rows, scale * 1.4426950408889634f,
                                   window, splits, status);
}

// copies the twelve ints that say where waits gave up last (see tc_attn_where)
int slb_prefill_attention_tc_where(int* out12) {
    return (int)cudaMemcpyFromSymbol(out12, tc_attn_where, 12 * sizeof(int));
}

int slb_prefill_attention_tc_status(int reset) {
    int v = 0;
    if (cudaMemcpyFromSymbol(&v, tc_attn_status, sizeof(int)) != cudaSuccess) return -1;
    if (reset && v != 0) {
        const int zero = 0;
        cudaMemcpyToSymbol(tc_attn_status, &zero, sizeof(int));
    }
    return v;
}
}

#else   // head sizes the tcgen05 kernel does not take

extern "C" {
int slb_prefill_attention_tc_supported(int, int) { return 0; }
int slb_prefill_attention_tc_tile_rows(int) { return 0; }
int slb_prefill_attention_tc_status(int) { return 0; }
int slb_prefill_attention_tc_where(int* out12) {
    for (int i = 0; i < 12; ++i) out12[i] = 0;
    return 0;
}
}

#endif

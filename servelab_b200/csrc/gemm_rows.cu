// Products of a feed-forward over the tokens of a prompt (or a portion of one) on the 5th-generation tensor cores,
// with what follows them in their epilogue:
//   gated    out[t, f] = act(x_t . Wg_f) (x_t . Wu_f), of one matrix or of one matrix an expert
//   experts  out[i, n] = x_i . W[e]_n, rows i of expert e (sorted by expert), bfloat16 or float32
// bfloat16 operands, float32 accumulation in tensor memory.  The gated form needs no gate|up matrix in memory and
// rounds the activation's result only.
//
// The rows of W are the M side of the MMA, 256 a pair of blocks (cta_group::2), the tokens its N side: a tile takes
// any multiple of 32 tokens up to 256, so that a step of any length, and an expert with any number of rows, is cut into
// tiles that fill the last wave.  A pair loads every operand once for both blocks: 128 rows of W and half of the token
// rows each.  What bounds a tile is the larger of its MMAs (2 nt cycles a k-block of 64: at nt = 256 one every 512
// cycles, measured 503) and its 256 + nt cycles of operands at the 64 bytes a cycle an SM takes from L2; a step of
// few tokens is bound by W's way from memory.
//
// Persistent blocks, one an SM: warp 0 loads (TMA tiles of 64 k through a ring of stages), warp 1 of the pair's first
// block issues the MMAs into one of two accumulators, warps 2..9 finish the other one meanwhile.  They transpose in
// registers: TMEM gives a thread one row of W and its tokens, memory wants neighbouring features of one token, so four
// lanes exchange four tokens (two shuffles for four values) and store 8 bytes each.
//
// Measured us, library product and activation -> this kernel (in a graph, weights not in L2): 0.5B shape, 65 / 257 /
// 480 / 1,000 / 2,048 tokens 8.2 / 11.5 / 14.3 / 22.4 / 39.2 -> 6.7 / 9.3 / 10.9 / 16.7 / 27.5; 7B shape, 128 / 480
// tokens 55 / 106 -> 45 / 96; experts' gate|up and down, 32 experts of 2,048 x 1,408, 4 of them a token, 64 / 512 /
// 2,048 tokens: library 134 / 138 / 176 -> 94 / 99 / 154.
//
// Every wait is bounded: after GR_SPIN_LIMIT polls a role sets the status word and leaves its loop; the
// loader waits (bounded) for its copies, the block frees its tensor memory and returns.
//
// Reference analogue: F.linear over a prompt (servelab/parallel/tp_model.py:48-53,67-68,115-119), left to
// the library there.
#include <cuda.h>

#include "gated_act.cuh"
#include "tma_util.cuh"

// 0, or (role << 8 | what) of the first wait that gave up
SLB_DEFINE_STATUS_WORD(gr_status_word, slb_gemm_rows_status)

namespace {

constexpr int GR_BM = 128;                 // rows of W a block
constexpr int GR_STEP = 32;                // tokens of a tile: a multiple of this
constexpr int GR_BK = 64;                  // k a stage: one 128-byte line of the swizzle
constexpr int GR_THREADS = 320;            // loader, MMA, eight epilogue warps
constexpr int GR_EPI_WARPS = 8;
constexpr int GR_MAX_STAGES = 12;
constexpr int GR_MAX_EXPERTS = 1024;
constexpr int GR_RUN = 64;                  // gates and ups alternating: rows of a run
constexpr int GR_MAX_TOKENS = 256;         // MMA N
constexpr int GR_W_BYTES = GR_BM * GR_BK * 2;
constexpr int GR_BAR_BYTES = 256;
constexpr size_t GR_SMEM_MAX = 227 * 1024;
constexpr size_t GR_PAIR_SMEM = 200 * 1024;
constexpr uint32_t GR_SPIN_LIMIT = 1u << 20;

enum { GR_STORE = 0, GR_GATED = 1, GR_F32 = 2 };     // bfloat16 rows, activation of gate and up, float32 rows

struct RowsArgs {
    void* out;                  // [T][ldo] bfloat16 (GR_F32: float)
    int ldo;
    int T, N, K;                // N: features of the result (GR_GATED: of the activation's)
    int nt;                     // tokens a tile (experts: at most)
    int w_tiles, tok_tiles;
    int stages, x_rows, x_box;  // x rows of a stage, per block, and of one copy
    int run;                    // GR_GATED: gates and ups of W alternate in runs of 64 rows (else: all gates, then all ups)
    const int* offsets;         // experts: rows of x before each, [E + 1]
    int E, w_expert_rows;
    float limit, alpha;
    const float* row_weights;   // GR_GATED, experts: weight of pair order[row], a factor on gate and up, or null
    const int* order;
    int acc_stride, acc_bufs, tmem_cols;
    int* status;
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
// bounded, entered by a whole warp: false in every lane if it ran out in one
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
    const uint32_t addr = smem_u32(bar);
    uint32_t done = 0;
    for (uint32_t i = 0; i < GR_SPIN_LIMIT && !done; ++i)
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done) : "r"(addr), "r"(parity) : "memory");
    return slb_warp_agrees(done != 0);
}
// the same word of shared memory in block `rank` of the cluster
__device__ __forceinline__ uint32_t in_block(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void arrive_at(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// a tile into this block's shared memory; its bytes are counted on a barrier of the pair's first block
__device__ __forceinline__ void load_tile(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
        "[%0], [%1, {%3, %4}], [%2];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1) : "memory");
}
// 64 gates and their ups (128 rows of W in the order of the epilogue's lanes) with one copy
__device__ __forceinline__ void load_gated_tile(uint32_t dst, const CUtensorMap* map, uint32_t bar, int k, int group, int outer) {
    asm volatile(
        "cp.async.bulk.tensor.5d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
        "[%0], [%1, {%3, %6, %6, %4, %5}], [%2];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(k), "r"(group), "r"(outer), "r"(0) : "memory");
}
// K-major operand tile, 128-byte swizzle: 8-row groups 1,024 bytes apart, descriptor version 1, layout 2
__device__ __forceinline__ uint64_t operand_desc(uint32_t smem_addr) {
    return (uint64_t)((smem_addr >> 4) & 0x3FFF) | (uint64_t)1 << 16 | (uint64_t)(1024 >> 4) << 32 | (uint64_t)1 << 46 |
           (uint64_t)2 << 61;
}
__device__ __forceinline__ void mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
// arrives at the barrier of both blocks when the MMAs issued so far are done
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(smem_u32(bar)), "h"((uint16_t)3) : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t addr, float (&v)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n\ttcgen05.wait::ld.sync.aligned;"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]),
          "=f"(v[8]), "=f"(v[9]), "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15]),
          "=f"(v[16]), "=f"(v[17]), "=f"(v[18]), "=f"(v[19]), "=f"(v[20]), "=f"(v[21]), "=f"(v[22]), "=f"(v[23]),
          "=f"(v[24]), "=f"(v[25]), "=f"(v[26]), "=f"(v[27]), "=f"(v[28]), "=f"(v[29]), "=f"(v[30]), "=f"(v[31])
        : "r"(addr) : "memory");
}
// 16 columns of the warp's 32 lanes; the values are there after tmem_wait
__device__ __forceinline__ void tmem_ld16(uint32_t addr, float (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]),
          "=f"(v[8]), "=f"(v[9]), "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15])
        : "r"(addr));
}
__device__ __forceinline__ void tmem_wait(float (&v)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+f"(v[0]), "+f"(v[1]), "+f"(v[2]), "+f"(v[3]), "+f"(v[4]), "+f"(v[5]), "+f"(v[6]), "+f"(v[7]),
                   "+f"(v[8]), "+f"(v[9]), "+f"(v[10]), "+f"(v[11]), "+f"(v[12]), "+f"(v[13]), "+f"(v[14]), "+f"(v[15])
                 :: "memory");
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
}
// Lane p of four neighbours has its own feature's values of tokens 0..3; afterwards it has token p's four
// features, as bfloat16.
__device__ __forceinline__ uint2 transpose4(float v0, float v1, float v2, float v3, int p) {
    const uint32_t w01 = pack_bf16(v0, v1), w23 = pack_bf16(v2, v3);
    const uint32_t got = __shfl_xor_sync(0xffffffffu, (p & 2) ? w01 : w23, 2);
    const uint32_t x = (p & 2) ? got : w01, y = (p & 2) ? w23 : got;       // features p & 1 and (p & 1) + 2
    const uint32_t lo = __byte_perm(x, y, 0x5410), hi = __byte_perm(x, y, 0x7632);
    const uint32_t keep = (p & 1) ? hi : lo, from = __shfl_xor_sync(0xffffffffu, (p & 1) ? lo : hi, 1);
    const uint32_t even = (p & 1) ? from : keep, odd = (p & 1) ? keep : from;
    return make_uint2(__byte_perm(even, odd, 0x5410), __byte_perm(even, odd, 0x7632));
}

struct Tile {
    int feat, matrix;           // this block's first feature, of which expert's matrix
    int tok, tok_end, nt;       // first token, end of the tile's tokens, MMA N
};

__host__ __device__ constexpr int gr_features(int epi) { return epi == GR_GATED ? GR_BM / 2 : GR_BM; }

// Tokens of an expert's tiles: as few tiles as fit, of equal size up to the rounding.
__device__ __forceinline__ int expert_tile_tokens(int n, int most) {
    const int c = (n + most - 1) / most;
    return c == 0 ? GR_STEP : ((n + c - 1) / c + GR_STEP - 1) / GR_STEP * GR_STEP;
}

// Tile `idx` for block `rank` of the pair.  Neighbouring tiles are token tiles of the same rows of W: a wave
// works on few rows of W, which are read from memory once.
template <int EPI, bool EXPERTS>
__device__ __forceinline__ Tile tile_of(const RowsArgs& a, const int* before, int idx, int rank) {
    Tile t;
    int w_tile;
    if (EXPERTS) {
        int lo = 0, hi = a.E;                              // before[lo] <= idx < before[hi]
        while (hi - lo > 1) {
            const int mid = (lo + hi) / 2;
            if (before[mid] <= idx) lo = mid; else hi = mid;
        }
        const int* offs = before + a.E + 1;
        const int r0 = offs[lo], r1 = offs[lo + 1], size = expert_tile_tokens(r1 - r0, a.nt);
        const int tiles = (r1 - r0 + size - 1) / size, local = idx - before[lo];
        w_tile = local / tiles;
        t.tok = r0 + (local - w_tile * tiles) * size;
        t.tok_end = min(r1, t.tok + size);
        t.nt = (t.tok_end - t.tok + GR_STEP - 1) / GR_STEP * GR_STEP;
        t.matrix = lo;
    } else {
        w_tile = idx / a.tok_tiles;
        t.tok = (idx - w_tile * a.tok_tiles) * a.nt;
        t.tok_end = min(a.T, t.tok + a.nt);
        t.nt = a.nt;
        t.matrix = 0;
    }
    t.feat = (w_tile * 2 + rank) * gr_features(EPI);
    return t;
}

template <int EPI, bool EXPERTS, int ACT>
__global__ void __launch_bounds__(GR_THREADS, 1) gemm_rows_kernel(const __grid_constant__ CUtensorMap map_w,
                                                                  const __grid_constant__ CUtensorMap map_x,
                                                                  const RowsArgs a) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* base = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
    const int x_bytes = a.x_rows * GR_BK * 2, stages = a.stages;
    unsigned char* x_stage = base + stages * GR_W_BYTES;
    uint64_t* full = reinterpret_cast<uint64_t*>(x_stage + stages * x_bytes);
    uint64_t* empty = full + GR_MAX_STAGES;
    uint64_t* acc_full = empty + GR_MAX_STAGES;
    uint64_t* acc_empty = acc_full + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
    int* before = reinterpret_cast<int*>(reinterpret_cast<unsigned char*>(full) + GR_BAR_BYTES);   // [E + 1], offsets [E + 1]

    const int warp = slb_warp(), lane = threadIdx.x & 31;
    uint32_t rank;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    const int first = blockIdx.x / 2, step = gridDim.x / 2, kblocks = (a.K + GR_BK - 1) / GR_BK;

    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], 2 * GR_EPI_WARPS);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(tmem_slot)), "r"(a.tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    int total = a.w_tiles * a.tok_tiles;
    if (EXPERTS) {
        pdl_wait();                                        // (the plan is a preceding kernel's)
        int* offs = before + a.E + 1;
        for (int e = threadIdx.x; e <= a.E; e += GR_THREADS) offs[e] = a.offsets[e];
        __syncthreads();
        if (warp == 0) {                                   // tiles before every expert
            int sum = 0;
            for (int e0 = 0; e0 < a.E; e0 += 32) {
                const int e = e0 + lane;
                const int n = e < a.E ? offs[e + 1] - offs[e] : 0, size = expert_tile_tokens(n, a.nt);
                int upto = (n + size - 1) / size * a.w_tiles;
                const int own = upto;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int v = __shfl_up_sync(0xffffffffu, upto, o);
                    if (lane >= o) upto += v;
                }
                if (e < a.E) before[e] = sum + upto - own;
                sum += __shfl_sync(0xffffffffu, upto, 31);
            }
            if (lane == 0) before[a.E] = sum;
        }
        __syncthreads();
        total = before[a.E];
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    cluster_sync();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;

    if (warp == 0) {
        // ------------------------------------------------------------ loader
        const uint32_t full0 = in_block(smem_u32(full), 0);
        const uint32_t w0 = smem_u32(base), x0 = smem_u32(x_stage);
        auto load_w = [&](const Tile& t, int kb, int s) {
            const uint32_t dst = w0 + s * GR_W_BYTES, bar = full0 + 8 * s;
            if (EPI == GR_GATED) {
                // 16 gates, their 16 ups, ...: a warp of the epilogue has both in its 32 rows
                if (a.run) load_gated_tile(dst, &map_w, bar, kb * GR_BK, 0, t.feat / GR_RUN);
                else load_gated_tile(dst, &map_w, bar, kb * GR_BK, t.feat / 16, t.matrix);
            } else {
                load_tile(dst, &map_w, bar, kb * GR_BK, t.matrix * a.w_expert_rows + t.feat);
            }
        };
        auto load_x = [&](const Tile& t, int kb, int s) {
            const uint32_t dst = x0 + s * x_bytes, bar = full0 + 8 * s;
            const int rows = t.nt / 2, r0 = t.tok + (int)rank * rows;
            if (EXPERTS)
                for (int r = 0; r < rows; r += a.x_box) load_tile(dst + r * 128, &map_x, bar, kb * GR_BK, r0 + r);
            else
                load_tile(dst, &map_x, bar, kb * GR_BK, r0);
        };
        auto expect = [&](const Tile& t, int s) {
            const int rows = EXPERTS ? (t.nt / 2 + a.x_box - 1) / a.x_box * a.x_box : t.nt / 2;
            if (rank == 0) mbar_expect_tx(&full[s], 2 * (GR_W_BYTES + rows * GR_BK * 2));
        };
        uint32_t it = 0;                                   // copies asked for
        int s = 0;                                         // stage, and the parity its next wait is for
        uint32_t phase = 1;
        bool ok = true;
        for (int idx = first; idx < total && ok; idx += step) {
            const Tile t = tile_of<EPI, EXPERTS>(a, before, idx, rank);
            int kb = 0;
            if (!EXPERTS && it == 0) {                     // W is written by no kernel: its first tiles need no wait
                const int ahead = min(kblocks, stages);
                for (int i = 0; i < ahead; ++i)
                    if (slb_elected()) {
                        expect(t, i);
                        load_w(t, i, i);
                    }
                pdl_wait();
                for (int i = 0; i < ahead; ++i)
                    if (slb_elected()) load_x(t, i, i);
                it = ahead;
                kb = ahead;
                s = ahead == stages ? 0 : ahead;
                phase = ahead == stages ? 0 : 1;
            }
            for (; kb < kblocks; ++kb, ++it) {
                if (!mbar_wait(&empty[s], phase)) {
                    atomicCAS(a.status, 0, (1 << 8) | 1);
                    ok = false;
                    break;
                }
                if (slb_elected()) {
                    expect(t, s);
                    load_w(t, kb, s);
                    load_x(t, kb, s);
                }
                if (++s == stages) {
                    s = 0;
                    phase ^= 1;
                }
            }
        }
        // (after a wait that gave up, the MMA issuer's as well, copies may be in flight; otherwise they have been waited for)
        if (rank == 0)
            for (uint32_t j = it > (uint32_t)stages ? it - stages : 0; j < it; ++j)
                mbar_wait(&full[j % stages], (j / stages) & 1);
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer (the pair's first block's)
        if (rank == 0) {
            pdl_wait();
            uint32_t n = 0, phase = 0;
            int s = 0;
            bool ok = true;
            const uint64_t w_desc = operand_desc(smem_u32(base)), x_desc = operand_desc(smem_u32(x_stage));
            for (int idx = first; idx < total && ok; idx += step, ++n) {
                const Tile t = tile_of<EPI, EXPERTS>(a, before, idx, 0);
                const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(t.nt >> 3) << 17) |
                                       ((uint32_t)(2 * GR_BM >> 4) << 24);
                const uint32_t buf = a.acc_bufs == 2 ? n & 1 : 0, use = a.acc_bufs == 2 ? n >> 1 : n;
                if (!mbar_wait(&acc_empty[buf], (use & 1) ^ 1)) {
                    atomicCAS(a.status, 0, (2 << 8) | 1);
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t acc = tmem + buf * a.acc_stride;
                for (int kb = 0; kb < kblocks; ++kb) {
                    if (!mbar_wait(&full[s], phase)) {
                        atomicCAS(a.status, 0, (2 << 8) | 2);
                        ok = false;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint64_t wd = w_desc + (uint64_t)(s * (GR_W_BYTES >> 4)), xd = x_desc + (uint64_t)(s * (x_bytes >> 4));
                    if (slb_elected()) {
#pragma unroll
                        for (int kk = 0; kk < GR_BK / 16; ++kk)
                            mma(acc, wd + 2 * kk, xd + 2 * kk, idesc, kb > 0 || kk > 0);
                        mma_commit(&empty[s]);
                        if (kb + 1 == kblocks) mma_commit(&acc_full[buf]);
                    }
                    if (++s == stages) {
                        s = 0;
                        phase ^= 1;
                    }
                }
            }
        }
    } else {
        // ------------------------------------------------------------ epilogue
        pdl_wait();
        const int quarter = warp & 3, half = (warp - 2) >> 2, p = lane & 3;
        const uint32_t empty0 = in_block(smem_u32(acc_empty), 0);
        bool released = false;
        uint32_t n = 0;
        for (int idx = first; idx < total; idx += step, ++n) {
            const Tile t = tile_of<EPI, EXPERTS>(a, before, idx, rank);
            const uint32_t buf = a.acc_bufs == 2 ? n & 1 : 0, use = a.acc_bufs == 2 ? n >> 1 : n;
            if (!mbar_wait(&acc_full[buf], use & 1)) {
                if (lane == 0) atomicCAS(a.status, 0, (3 << 8) | 1);
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (!released && idx + step >= total) {
                pdl_launch_dependents();
                released = true;
            }
            const uint32_t acc = tmem + buf * a.acc_stride + ((uint32_t)(quarter * 32) << 16);
            const int tokens = t.tok_end - t.tok;
            const int f = t.feat + (EPI == GR_GATED ? quarter * 16 + (lane & 15) : quarter * 32 + lane);
            const int f4 = f & ~3;
            if constexpr (EPI == GR_GATED) {
                // 16 tokens at a time, the next ones on their way from tensor memory.  (A short loop: unrolled over
                // a tile a launch took 6 us more.)
                const int up = lane >> 4;                  // lanes 0..15 hold gates, the others their ups
                float v[16], next[16];
                if (half * 16 < tokens) {
                    tmem_ld16(acc + half * 16, v);
                    tmem_wait(v);
                }
#pragma unroll 1
                for (int c = half * 16; c < tokens; c += 32) {
                    const bool more = c + 32 < tokens;
                    if (more) tmem_ld16(acc + c + 32, next);
                    float r[8];                            // tokens c + 2 m + up
#pragma unroll
                    for (int m = 0; m < 8; ++m) {
                        const float got = __shfl_xor_sync(0xffffffffu, up ? v[2 * m] : v[2 * m + 1], 16);
                        float gv = up ? got : v[2 * m], uv = up ? v[2 * m + 1] : got;
                        if (EXPERTS && a.row_weights != nullptr) {
                            const int row = t.tok + c + 2 * m + up;
                            const float wt = row < t.tok_end ? a.row_weights[a.order[row]] : 0.f;
                            gv *= wt;
                            uv *= wt;
                        }
                        r[m] = act_mul_sums<ACT>(gv, uv, a.limit, a.alpha);
                    }
                    bf16* dst = static_cast<bf16*>(a.out) + (size_t)(t.tok + c + 2 * p + up) * a.ldo + f4;
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const uint2 w = transpose4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3], p);
                        if (c + 8 * j + 2 * p + up < tokens && f4 < a.N)
                            *reinterpret_cast<uint2*>(dst + (size_t)(8 * j) * a.ldo) = w;
                    }
                    if (more) {
                        tmem_wait(next);
#pragma unroll
                        for (int j = 0; j < 16; ++j) v[j] = next[j];
                    }
                }
            } else {
#pragma unroll 1
                for (int c = half * 32; c < tokens; c += 64) {
                    float v[32];
                    tmem_ld32(acc + c, v);
                    if (EPI == GR_F32) {
                        float* dst = static_cast<float*>(a.out) + (size_t)(t.tok + c) * a.ldo + f;
                        if (f < a.N) {
#pragma unroll
                            for (int j = 0; j < 32; ++j)
                                if (c + j < tokens) dst[(size_t)j * a.ldo] = v[j];
                        }
                    } else {
                        bf16* dst = static_cast<bf16*>(a.out) + (size_t)(t.tok + c + p) * a.ldo + f4;
#pragma unroll
                        for (int j = 0; j < 32; j += 4) {
                            const uint2 w = transpose4(v[j], v[j + 1], v[j + 2], v[j + 3], p);
                            if (c + j + p < tokens && f4 < a.N) *reinterpret_cast<uint2*>(dst + (size_t)j * a.ldo) = w;
                        }
                    }
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) arrive_at(empty0 + 8 * buf);
        }
    }
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    cluster_sync();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(a.tmem_cols) : "memory");
    }
}

// boxes of `box_rows` x 64 of a row-major bfloat16 matrix [rows, K], 128-byte swizzle, zeros outside
int rows_map(CUtensorMap* map, const void* ptr, long long rows, int K, int ld, int box_rows) {
    slb_tma::EncodeTiledFn fn = slb_tma::encode_tiled();
    if (fn == nullptr) return SLB_ERR_BAD_ARG;
    const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
    const cuuint32_t box[2] = {(cuuint32_t)GR_BK, (cuuint32_t)box_rows};
    const cuuint32_t elem[2] = {1, 1};
    const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, elem,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : SLB_ERR_BAD_ARG;
}

// W of a gated product with gate f, up f as rows (f / 64) * 128 + f % 64 and 64 further (run), or f and I further, as
// [outer][group of 16 features][gate, up][16 rows][K]; `I` a multiple of 16 (run: of 64).  outer: runs or matrices.
int gated_map(CUtensorMap* map, const void* ptr, int K, int ld, int I, int run, int matrices) {
    slb_tma::EncodeTiledFn fn = slb_tma::encode_tiled();
    if (fn == nullptr) return SLB_ERR_BAD_ARG;
    const cuuint64_t row = (cuuint64_t)ld * 2;
    const cuuint64_t dims[5] = {(cuuint64_t)K, 16, 2, (cuuint64_t)(run ? GR_RUN / 16 : I / 16),
                                (cuuint64_t)(run ? I / GR_RUN : matrices)};
    const cuuint64_t strides[4] = {row, row * (run ? GR_RUN : I), row * 16, row * 2 * (run ? GR_RUN : I)};
    const cuuint32_t box[5] = {(cuuint32_t)GR_BK, 16, 2, 4, 1};
    const cuuint32_t elem[5] = {1, 1, 1, 1, 1};
    const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<void*>(ptr), dims, strides, box, elem,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : SLB_ERR_BAD_ARG;
}

// Tokens a tile for T tokens: the fewest cycles of rounds x (256 + nt) a k-block, and the last tile's epilogue (22 a
// token).  Measured us at 160 / 192 / 224 / 256 a tile: 480 tokens of the 0.5B shape 10.9 / 11.4 / - / 13.4, 1,000 17.5 /
// 17.7 / 16.7 / -, 2,048 29.4 / 28.0 / 28.7 / 27.5; 2,048 tokens of 2,048 x 5,632 35.2 / 35.6 / 34.5 / 36.6: the rule
// takes the least each time.
int tile_tokens(int T, int w_tiles, int K, int pairs) {
    long long best = 0;
    int nt = 0;
    for (int n = GR_STEP; n <= GR_MAX_TOKENS; n += GR_STEP) {
        const long long tiles = (long long)w_tiles * ((T + n - 1) / n), rounds = (tiles + pairs - 1) / pairs;
        const long long cycles = rounds * ((K + GR_BK - 1) / GR_BK) * (256 + n) + 22 * n;
        if (nt == 0 || cycles < best) {
            best = cycles;
            nt = n;
        }
    }
    return nt;
}

template <int EPI, bool EXPERTS, int ACT = 0>
int launch_rows(const bf16* x, int ldx, const bf16* W, int ldw, RowsArgs a, cudaStream_t st) {
    const int pairs = slb_num_sms() / 2;
    a.w_tiles = (a.N + 2 * gr_features(EPI) - 1) / (2 * gr_features(EPI));
    long long tiles = 1ll << 30;
    if (!EXPERTS) {
        if (a.nt == 0) a.nt = tile_tokens(a.T, a.w_tiles, a.K, pairs);
        a.tok_tiles = (a.T + a.nt - 1) / a.nt;
        tiles = (long long)a.w_tiles * a.tok_tiles;
        if (tiles > 1 << 30) return SLB_ERR_TOO_LARGE;
    }
    const int groups = (int)(tiles < pairs ? tiles : pairs);
    // (experts: a crowded one's rows in small tiles where the large ones would leave most pairs without any)
    if (EXPERTS) a.nt = (long long)a.w_tiles * (a.T / GR_MAX_TOKENS + a.E) < pairs ? 64 : GR_MAX_TOKENS;
    a.x_rows = a.nt / 2;
    // (experts: copies as tall as an expert's share, so that few are issued and few rows are brought in vain)
    a.x_box = !EXPERTS ? a.x_rows : a.T <= 32 * a.E ? 16 : a.T <= 64 * a.E || a.nt == 64 ? 32 : 64;
    a.acc_stride = a.nt;
    a.acc_bufs = tiles > groups ? 2 : 1;
    a.tmem_cols = 32;
    while (a.tmem_cols < a.acc_stride * a.acc_bufs) a.tmem_cols *= 2;
    const size_t stage = GR_W_BYTES + (size_t)a.x_rows * GR_BK * 2;
    const size_t tail = GR_BAR_BYTES + (EXPERTS ? (size_t)(2 * (a.E + 1) + 3) / 4 * 16 : 0);
    a.stages = (int)((GR_SMEM_MAX - 1024 - tail) / stage);
    if (a.stages > GR_MAX_STAGES) a.stages = GR_MAX_STAGES;
    CUtensorMap map_w, map_x;
    int rc = EPI == GR_GATED ? gated_map(&map_w, W, a.K, ldw, a.N, a.run, EXPERTS ? a.E : 1)
                             : rows_map(&map_w, W, (long long)a.E * a.w_expert_rows, a.K, ldw, GR_BM);
    if (rc == 0) rc = rows_map(&map_x, x, a.T, a.K, ldx, a.x_box);
    if (rc != 0) return rc;
    static unsigned long long configured = 0;
    rc = slb_configure(&configured, gemm_rows_kernel<EPI, EXPERTS, ACT>, GR_SMEM_MAX);
    if (rc != 0) return rc;
    const cudaError_t e = cudaGetSymbolAddress((void**)&a.status, gr_status_word);
    if (e != cudaSuccess) return (int)e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(groups * 2);
    cfg.blockDim = dim3(GR_THREADS);
    // A pair allocates its tensor memory on two SMs at once: it keeps each to itself (no other kernel with
    // tensor memory fits beside 200 KB), so that no two allocations can wait for each other's half.
    const size_t smem = 1024 + a.stages * stage + tail;
    cfg.dynamicSmemBytes = smem > GR_PAIR_SMEM ? smem : GR_PAIR_SMEM;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = slb_pdl_enabled ? 2 : 1;
    return (int)cudaLaunchKernelEx(&cfg, gemm_rows_kernel<EPI, EXPERTS, ACT>, map_w, map_x, (const RowsArgs)a);
}
template <bool EXPERTS>
int launch_gated(int act, const bf16* x, int ldx, const bf16* W, int ldw, const RowsArgs& a, cudaStream_t st) {
    if (act == 0) return launch_rows<GR_GATED, EXPERTS, 0>(x, ldx, W, ldw, a, st);
    if (act == 1) return launch_rows<GR_GATED, EXPERTS, 1>(x, ldx, W, ldw, a, st);
    if (act == 2 && a.limit > 0.f) return launch_rows<GR_GATED, EXPERTS, 2>(x, ldx, W, ldw, a, st);
    return SLB_ERR_BAD_ARG;
}

int check_operands(const bf16* x, int ldx, const bf16* W, int ldw, int K) {
    if (K <= 0 || K % 8 || ldw % 8 || ldw < K || (uintptr_t)W % 16 || W == nullptr) return SLB_ERR_BAD_ARG;
    if (x == nullptr || ldx % 8 || ldx < K || (uintptr_t)x % 16) return SLB_ERR_BAD_ARG;
    return 0;
}
int check_out(const void* out, int ldo, int N) {
    return out == nullptr || (uintptr_t)out % 8 || ldo % 4 || N <= 0 || N % 4 || ldo < N ? SLB_ERR_BAD_ARG : 0;
}

}  // namespace

extern "C" {

// out[T, I] = act(x Wg^T) (x Wu^T); W [2 I, K]: gates then ups (run = 0; I a multiple of 16), or alternating in runs
// of 64 rows (run = 64; I a multiple of 64).  act, limit, alpha as in gated_act.cuh.  nt: tokens a tile (a multiple of 32
// up to 256), 0: by the rule above.
int slb_gemm_rows_gated_bf16(const bf16* x, int ldx, const bf16* W, int ldw, bf16* out, int ldo, int T, int I, int K,
                             int run, int act, float limit, float alpha, int nt, cudaStream_t st) {
    if (T == 0) return 0;
    int rc = check_operands(x, ldx, W, ldw, K);
    if (rc == 0) rc = check_out(out, ldo, I);
    if (rc != 0 || T < 0 || (run != 0 && run != GR_RUN) || I % (run ? GR_RUN : 16) || nt < 0 || nt > GR_MAX_TOKENS ||
        nt % GR_STEP)
        return rc != 0 ? rc : SLB_ERR_BAD_ARG;
    if (I > 1 << 29) return SLB_ERR_TOO_LARGE;
    RowsArgs a = {};
    a.out = out; a.ldo = ldo; a.T = T; a.N = I; a.K = K; a.nt = nt;
    a.run = run; a.limit = limit; a.alpha = alpha;
    return launch_gated<false>(act, x, ldx, W, ldw, a, st);
}

// Experts: rows offsets[e] .. offsets[e + 1] of x [P, K] and out belong to expert e (rows of none are not written); W
// [E][rows][K].  gated: rows = 2 N, gates then ups (N a multiple of 16); row_weights / order: row i's gate and up times
// row_weights[order[i]].  out_f32: float32 rows (not gated).
int slb_gemm_rows_experts_bf16(const bf16* x, int ldx, const bf16* W, int ldw, void* out, int ldo, const int* offsets,
                               int E, int P, int N, int K, int gated, int out_f32, int act, float limit, float alpha,
                               const float* row_weights, const int* order, cudaStream_t st) {
    if (P == 0) return 0;
    int rc = check_operands(x, ldx, W, ldw, K);
    if (rc == 0) rc = check_out(out, ldo, N);
    if (rc != 0 || P < 0 || E <= 0 || offsets == nullptr) return rc != 0 ? rc : SLB_ERR_BAD_ARG;
    if (E > GR_MAX_EXPERTS || N > 1 << 29) return SLB_ERR_TOO_LARGE;
    if (gated && (N % 16 || out_f32)) return SLB_ERR_BAD_ARG;
    if (row_weights != nullptr && (order == nullptr || !gated)) return SLB_ERR_BAD_ARG;
    RowsArgs a = {};
    a.out = out; a.ldo = ldo; a.T = P; a.N = N; a.K = K;
    a.offsets = offsets; a.E = E; a.w_expert_rows = gated ? 2 * N : N;
    a.limit = limit; a.alpha = alpha; a.row_weights = row_weights; a.order = order;
    if ((long long)E * a.w_expert_rows > 1 << 30) return SLB_ERR_TOO_LARGE;
    if (gated) return launch_gated<true>(act, x, ldx, W, ldw, a, st);
    return out_f32 ? launch_rows<GR_F32, true>(x, ldx, W, ldw, a, st) : launch_rows<GR_STORE, true>(x, ldx, W, ldw, a, st);
}

}  // extern "C"

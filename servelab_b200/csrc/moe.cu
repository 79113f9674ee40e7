// Routed experts: the router's choice, the plan of a step (which rows each expert gets), the
// experts' products on CUDA cores, and the weighted sum.
//
//   slb_moe_route      scores = softmax(logits) in float32 per token; experts form `groups` equal
//                      groups of neighbours, a group's score is its largest score, only experts of
//                      the `keep` best groups can be chosen; the `top` largest scores among those
//                      are the choice (ties: the lower index); weight = score * route_scale
//                      (optionally divided by the sum of the chosen scores).
//   slb_moe_route_scored  the same with sigmoid scores, an offset per expert that enters the choice
//                      only, groups that score as the sum of their best few, and a constant in the
//                      denominator of the renormalised weights, each an argument.
//   slb_moe_plan(_simt)  (token, choice) pairs sorted by expert: counts, offsets, the list, and the
//                      row tiles of the products (tile -> expert, first row), of a length that
//                      depends only on the number of pairs and experts (a fixed grid).
//   slb_moe_gate_up    act[pair] = silu(W_gate[e] x) * (W_up[e] x) for the pair's expert e, or another gated
//                      activation; with `in_weights` the expert's input is the pair's weight times x
//                      (a factor on both sums, since the products are linear);
//   slb_moe_down       y[pair] = W_down[e] act[pair], float32;
//   slb_moe_combine    out[t] = (shared[t]) + sum_k weight[t][k] * y[t * top + k], in the order k (no
//                      weights: the plain sum).
//
// Each output element of a product is a sum over k = 0..K-1 in that order (plain FFMA), and the
// combine adds a token's experts in the order of its choice, so a token's result does not depend
// on what else is in the batch.
#include "gated_act.cuh"
#include "mma_util.cuh"

#define MOE_MAX_EXPERTS 1024
#define MOE_MAX_TOP 32
#define MOE_BM 64
#define MOE_BN 64
#define MOE_BK 16

// Rows of a tile of the tensor-core product: few where an expert gets few, so that its stages are small and
// all its blocks are resident at once (the last wave of a second round is nearly empty).  The product on CUDA
// cores has tiles of MOE_BM rows whatever they hold: a smaller one would cost it as much.
// The line at 32 rows an expert, us of a step with tiles of 32 / 64 rows at 28, 36, 44 rows each: 128 experts of
// 2,048 x 768 313 / 293, 398 / 323, 460 / 353; 32 of 2,048 x 1,408 149 / 185, 206 / 189, 230 / 195; 64 of
// 1,024 x 512 79 / 71, 94 / 77, 106 / 83.  With few experts there are too few tiles to fill the device and the
// smaller ones stay ahead for longer, at 36, 50, 64: 16 of 1,024 x 512 38 / 47, 40 / 49, 44 / 54; 8 of 2,048 x 1,408
// 76 / 86, 80 / 98, 82 / 101.
static int moe_tile_rows(int P, int E) { return P <= 8 * E ? 16 : P <= (E <= 16 ? 64 : 32) * E ? 32 : MOE_BM; }
static int moe_num_tiles(int P, int E, int rows) { return (P + rows - 1) / rows + E; }
static int moe_num_tiles(int P, int E) { return moe_num_tiles(P, E, moe_tile_rows(P, E)); }
static int moe_plan_ints(int P, int E, int rows) { return 3 * E + 1 + 2 * moe_num_tiles(P, E, rows) + 2 * P; }

// ------------------------------------------------------------------- route
__device__ __forceinline__ void warp_argmax(float& v, int& i) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, v, o);
        const int oi = __shfl_xor_sync(0xffffffffu, i, o);
        if (ov > v || (ov == v && oi < i)) {
            v = ov;
            i = oi;
        }
    }
}

// One warp a token.  `score_fn` 0: scores = softmax(logits); 1: scores = sigmoid(logits).  The
// choice runs on choice scores c = score (+ correction[e], a learned offset that enters the choice
// only; sigmoids without offset and groups: c = the logit); a group's score is the sum of its `group_best` largest choice scores (1: its maximum);
// experts outside the `keep` best groups count as minus infinity (choice scores may be negative);
// the weights are the chosen experts' scores without the offset, divided by their sum + `norm_eps`
// with `renormalize`, times `route_scale`.  Ties: the lower index.
__global__ void __launch_bounds__(128) moe_route_kernel(
    const float* __restrict__ logits, int ldl, int T, int E, int groups, int keep, int top,
    float route_scale, int renormalize, int score_fn, const float* __restrict__ correction, int group_best,
    float norm_eps, int* __restrict__ ids, float* __restrict__ weights) {
    extern __shared__ float route_smem[];
    pdl_wait();
    pdl_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t = blockIdx.x * 4 + warp;
    if (t >= T) return;
    float* s = route_smem + (size_t)warp * (2 * E + 2 * groups);   // scores, choice scores,
    float* c = s + E;                                                // the groups' scores and marks
    float* gs = c + E;
    float* gmark = gs + groups;
    const float* z = logits + (size_t)t * ldl;
    if (score_fn == 0) {
        float mx = -INFINITY;
        for (int e = lane; e < E; e += 32) mx = fmaxf(mx, z[e]);
        mx = warp_max(mx);
        float sum = 0.f;
        for (int e = lane; e < E; e += 32) {
            const float p = expf(z[e] - mx);
            s[e] = p;
            sum += p;
        }
        sum = warp_sum(sum);
        const float inv = 1.0f / sum;
        for (int e = lane; e < E; e += 32) s[e] *= inv;
    } else {
        for (int e = lane; e < E; e += 32) s[e] = 1.0f / (1.0f + expf(-z[e]));
    }
    __syncwarp();
    // (sigmoids alone: the logits give the same order, also where their sigmoids round to the same number)
    const bool by_logit = score_fn == 1 && correction == nullptr && groups == 1;
    for (int e = lane; e < E; e += 32) c[e] = by_logit ? z[e] : correction != nullptr ? s[e] + correction[e] : s[e];
    __syncwarp();
    const int per = E / groups;
    if (groups > 1) {
        for (int g = lane; g < groups; g += 32) {
            // the sum of the group's `group_best` largest choice scores (all of them if it has fewer)
            float total = 0.f;
            int prev_i = -1;
            float prev_v = INFINITY;
            const int take = group_best < per ? group_best : per;
            for (int r = 0; r < take; ++r) {
                float b = -INFINITY;
                int bi = -1;
                for (int e = g * per; e < (g + 1) * per; ++e) {
                    const float v = c[e];
                    const bool after = v < prev_v || (v == prev_v && e > prev_i);   // not yet taken
                    if (after && (bi < 0 || v > b)) {
                        b = v;
                        bi = e;
                    }
                }
                if (bi < 0) break;
                total += b;
                prev_v = b;
                prev_i = bi;
            }
            gs[g] = total;
            gmark[g] = 0.f;
        }
        __syncwarp();
        for (int round = 0; round < keep; ++round) {
            float bv = -INFINITY;
            int bi = 0x7fffffff;
            for (int g = lane; g < groups; g += 32)
                if (gmark[g] == 0.f && (gs[g] > bv || (gs[g] == bv && g < bi) || bi == 0x7fffffff) && gs[g] == gs[g]) {
                    bv = gs[g];
                    bi = g;
                }
            warp_argmax(bv, bi);
            if (lane == 0 && bi < groups) gmark[bi] = 1.f;   // (no group found: logits that are no numbers)
            __syncwarp();
        }
        for (int e = lane; e < E; e += 32)
            if (gmark[e / per] == 0.f) c[e] = -INFINITY;
        __syncwarp();
    }
    float chosen_sum = 0.f;
    for (int round = 0; round < top; ++round) {
        float bv = -INFINITY;
        int bi = 0x7fffffff;
        for (int e = lane; e < E; e += 32) {
            const float v = c[e];
            if (v > -INFINITY && (v > bv || (v == bv && e < bi) || bi == 0x7fffffff)) {
                bv = v;
                bi = e;
            }
        }
        warp_argmax(bv, bi);
        float w = 0.f;
        if (bi >= E) {                                     // nothing left to choose (logits that are no
            bi = 0;                                        // numbers, as the rows of a padded step may
        } else {                                           // hold): expert 0 with weight 0
            w = s[bi];
        }
        __syncwarp();
        if (lane == 0) {
            ids[(size_t)t * top + round] = bi;
            weights[(size_t)t * top + round] = w;
            if (w == w && c[bi] > -INFINITY) c[bi] = -INFINITY;      // taken
        }
        chosen_sum += w;
        __syncwarp();
    }
    if (lane < top) {
        float w = weights[(size_t)t * top + lane];
        if (renormalize) w /= (chosen_sum + norm_eps);
        weights[(size_t)t * top + lane] = w * route_scale;
    }
}

// The same for up to 128 experts in at most 32 groups that score as their best expert: a lane holds the scores of
// experts lane, lane + 32, ...; a choice is the largest of 32 unsigned keys in the order of the scores (0: not to be
// chosen), found by the warp's reduction instruction, then the lowest index that has it.  The sums are those of the
// kernel above.  What bounds either is one warp's chain of reductions: us, kernel above / this one: 4 of 32 experts in
// 2 of 4 groups, 64 tokens 5.1 / 2.4, 2,048 6.1 / 3.1; 8 of 128, 64 tokens 6.5 / 2.3, 2,048 7.6 / 3.3.
#define MOE_FEW_EXPERTS 128
__device__ __forceinline__ unsigned score_key(float v) {
    const unsigned b = __float_as_uint(v + 0.0f);              // (both zeros are one)
    return v > -INFINITY ? b ^ ((b >> 31) ? 0xffffffffu : 0x80000000u) : 0u;     // (no number: 0)
}
__global__ void __launch_bounds__(128) moe_route_few_kernel(
    const float* __restrict__ logits, int ldl, int T, int E, int groups, int keep, int top, float route_scale,
    int renormalize, int score_fn, const float* __restrict__ correction, float norm_eps, int* __restrict__ ids,
    float* __restrict__ weights) {
    constexpr int PER = MOE_FEW_EXPERTS / 32;
    __shared__ float choice[4][MOE_FEW_EXPERTS];
    pdl_wait();
    pdl_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t = blockIdx.x * 4 + warp;
    if (t >= T) return;
    const float* z = logits + (size_t)t * ldl;
    float l[PER], s[PER], c[PER];
#pragma unroll
    for (int j = 0; j < PER; ++j) l[j] = lane + 32 * j < E ? z[lane + 32 * j] : -INFINITY;
    if (score_fn == 0) {
        float mx = -INFINITY, sum = 0.f;
#pragma unroll
        for (int j = 0; j < PER; ++j) mx = fmaxf(mx, l[j]);
        mx = warp_max(mx);
#pragma unroll
        for (int j = 0; j < PER; ++j) {
            s[j] = 0.f;
            if (lane + 32 * j < E) sum += s[j] = expf(l[j] - mx);
        }
        const float inv = 1.0f / warp_sum(sum);
#pragma unroll
        for (int j = 0; j < PER; ++j) s[j] *= inv;
    } else {
#pragma unroll
        for (int j = 0; j < PER; ++j) s[j] = 1.0f / (1.0f + expf(-l[j]));
    }
    const bool by_logit = score_fn == 1 && correction == nullptr && groups == 1;
    unsigned key[PER];
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        const int e = lane + 32 * j;
        c[j] = by_logit ? l[j] : correction != nullptr && e < E ? s[j] + correction[e] : s[j];
        key[j] = e < E ? score_key(c[j]) : 0u;
    }
    if (groups > 1) {
        const int per = E / groups;
#pragma unroll
        for (int j = 0; j < PER; ++j)
            if (lane + 32 * j < E) choice[warp][lane + 32 * j] = c[j];
        __syncwarp();
        // a group's score: its best choice score (0 where none is a number)
        float best = -INFINITY;
        bool any = false;
        if (lane < groups)
            for (int i = 0; i < per; ++i) {
                const float v = choice[warp][lane * per + i];
                any = any || v == v;
                best = fmaxf(best, v);
            }
        best = any ? best : 0.f;
        // (a group of minus infinities can still be kept where fewer others are there: key 1, below every number's)
        unsigned group_key = lane < groups ? max(score_key(best), 1u) : 0u, kept = 0u;
        for (int round = 0; round < keep; ++round) {
            const unsigned m = __reduce_max_sync(0xffffffffu, group_key);
            if (m == 0u) break;
            const int g = __ffs(__ballot_sync(0xffffffffu, group_key == m)) - 1;
            kept |= 1u << g;
            if (lane == g) group_key = 0u;
        }
#pragma unroll
        for (int j = 0; j < PER; ++j) {
            const int e = lane + 32 * j;
            if (e < E && !(kept >> (e / per) & 1u)) key[j] = 0u;
        }
    }
    float chosen_sum = 0.f, my_weight = 0.f;
    int my_id = 0;
    for (int round = 0; round < top; ++round) {
        unsigned m = key[0];
#pragma unroll
        for (int j = 1; j < PER; ++j) m = max(m, key[j]);
        m = __reduce_max_sync(0xffffffffu, m);
        int e = 0x7fffffff;
#pragma unroll
        for (int j = PER - 1; j >= 0; --j)
            if (m != 0u && key[j] == m) e = lane + 32 * j;
        e = __reduce_min_sync(0xffffffffu, e);
        float w = 0.f;
        if (e < E) {
            float mine = 0.f;
#pragma unroll
            for (int j = 0; j < PER; ++j)
                if (lane + 32 * j == e) {
                    mine = s[j];
                    if (mine == mine) key[j] = 0u;             // taken
                }
            w = __shfl_sync(0xffffffffu, mine, e & 31);
        } else {
            e = 0;                                             // nothing left to choose: expert 0 with weight 0
        }
        if (lane == round) {
            my_id = e;
            my_weight = w;
        }
        chosen_sum += w;
    }
    if (lane < top) {
        ids[(size_t)t * top + lane] = my_id;
        weights[(size_t)t * top + lane] = (renormalize ? my_weight / (chosen_sum + norm_eps) : my_weight) * route_scale;
    }
}

// ----------------------------------------------------------- router logits
// logits[t][e] = sum_k x[t][k] * w[e][k] in float32 (w float32, x float32 or bfloat16).  A block
// owns ROUTER_TOK tokens and one expert; its eight warps take an eighth of k each (lanes stride,
// coalesced) and the partial sums are added in a fixed order, so a token's logits do not depend
// on the batch.
#define ROUTER_TOK 4
template <typename T>
__global__ void __launch_bounds__(256) router_logits_kernel(const T* __restrict__ x, int ldx,
                                                            const float* __restrict__ w, int ldw,
                                                            float* __restrict__ logits, int ldl, int M,
                                                            int E, int K) {
    __shared__ float part[8][ROUTER_TOK];
    pdl_wait();
    pdl_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t0 = blockIdx.x * ROUTER_TOK;
    const int e = blockIdx.y;
    const T* xr[ROUTER_TOK];
#pragma unroll
    for (int i = 0; i < ROUTER_TOK; ++i) xr[i] = x + (size_t)min(t0 + i, M - 1) * ldx;
    const float* wr = w + (size_t)e * ldw;
    const int per = (K + 7) / 8;
    const int k_end = min(K, (warp + 1) * per);
    float acc[ROUTER_TOK];
#pragma unroll
    for (int i = 0; i < ROUTER_TOK; ++i) acc[i] = 0.f;
#pragma unroll 4
    for (int k = warp * per + lane; k < k_end; k += 32) {
        const float wv = wr[k];
#pragma unroll
        for (int i = 0; i < ROUTER_TOK; ++i) acc[i] = fmaf(to_float(xr[i][k]), wv, acc[i]);
    }
#pragma unroll
    for (int i = 0; i < ROUTER_TOK; ++i) {
        const float v = warp_sum(acc[i]);
        if (lane == 0) part[warp][i] = v;
    }
    __syncthreads();
    if (threadIdx.x < ROUTER_TOK && t0 + threadIdx.x < M) {
        float v = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) v += part[j][threadIdx.x];
        logits[(size_t)(t0 + threadIdx.x) * ldl + e] = v;
    }
}

// The same for steps of many tokens: a block owns 16 tokens and 32 experts, its eight warps an eighth of k
// each, brought in by cp.async through a ring of the warp's own (no block-wide wait); a lane sums 4 tokens by
// 4 experts in float32, the warps' sums are added in order.  What bounds it is the FFMA issue of the few
// blocks and the router's matrix, which every block reads from L2.
#define RL_TOK 16
#define RL_EXP 32
#define RL_KC 32
#define RL_STAGES 3
struct __align__(16) RouterStage {
    bf16 x[RL_TOK][RL_KC + 8];
    float w[RL_EXP][RL_KC + 4];
};
__global__ void __launch_bounds__(256) router_logits_tile_kernel(const bf16* __restrict__ x, int ldx,
                                                                 const float* __restrict__ w, int ldw,
                                                                 float* __restrict__ logits, int ldl, int M, int E,
                                                                 int K) {
    using namespace slb_mma;
    extern __shared__ __align__(16) unsigned char rl_smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    RouterStage* ring = reinterpret_cast<RouterStage*>(rl_smem) + warp * RL_STAGES;
    const int t0 = blockIdx.x * RL_TOK, e0 = blockIdx.y * RL_EXP;
    const int chunks = K / RL_KC, first = warp * chunks / 8, mine = (warp + 1) * chunks / 8 - first;
    pdl_wait();
    pdl_launch_dependents();
    auto fetch = [&](int i) {
        RouterStage& st = ring[i % RL_STAGES];
        const int k0 = (first + i) * RL_KC;
#pragma unroll
        for (int q = 0; q < 2; ++q) {                     // 16 rows of 4 pieces
            const int p = lane + q * 32, r = p >> 2, c = (p & 3) * 8;
            const bool ok = t0 + r < M;
            cp_async16(&st.x[r][c], x + (size_t)(ok ? t0 + r : 0) * ldx + k0 + c, ok);
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) {                     // 32 rows of 8 pieces
            const int p = lane + q * 32, r = p >> 3, c = (p & 7) * 4;
            const bool ok = e0 + r < E;
            cp_async16(&st.w[r][c], w + (size_t)(ok ? e0 + r : 0) * ldw + k0 + c, ok);
        }
    };
#pragma unroll
    for (int i = 0; i < RL_STAGES - 1; ++i) {
        if (i < mine) fetch(i);
        cp_async_commit();
    }
    const int ty = lane >> 3, tx = lane & 7;              // tokens ty + 4 i, experts tx + 8 j
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
    for (int c = 0; c < mine; ++c) {
        cp_async_wait<RL_STAGES - 2>();
        __syncwarp();                                     // chunk c is there; chunk c - 1 has been read
        if (c + RL_STAGES - 1 < mine) fetch(c + RL_STAGES - 1);
        cp_async_commit();
        const RouterStage& st = ring[c % RL_STAGES];
#pragma unroll
        for (int k = 0; k < RL_KC; k += 4) {
            float xv[4][4], wv[4][4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint2 r = *reinterpret_cast<const uint2*>(&st.x[ty + 4 * i][k]);
                xv[i][0] = __uint_as_float(r.x << 16);
                xv[i][1] = __uint_as_float(r.x & 0xffff0000u);
                xv[i][2] = __uint_as_float(r.y << 16);
                xv[i][3] = __uint_as_float(r.y & 0xffff0000u);
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float4 r = *reinterpret_cast<const float4*>(&st.w[tx + 8 * j][k]);
                wv[j][0] = r.x; wv[j][1] = r.y; wv[j][2] = r.z; wv[j][3] = r.w;
            }
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(xv[i][kk], wv[j][kk], acc[i][j]);
        }
    }
    cp_async_wait<0>();
    __syncthreads();                                      // the rings are free: the warps' sums take their place
    float* part = reinterpret_cast<float*>(rl_smem);      // [8][RL_TOK][RL_EXP]
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) part[(warp * RL_TOK + ty + 4 * i) * RL_EXP + tx + 8 * j] = acc[i][j];
    __syncthreads();
    for (int o = threadIdx.x; o < RL_TOK * RL_EXP; o += 256) {
        const int t = t0 + o / RL_EXP, e = e0 + o % RL_EXP;
        float v = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) v += part[i * RL_TOK * RL_EXP + o];
        if (t < M && e < E) logits[(size_t)t * ldl + e] = v;
    }
}

// -------------------------------------------------------------------- plan
// One block.  plan = [counts E | offsets E + 1 | unused E | tile_expert NT | tile_row0 NT |
// sorted P | where P] (int32), NT = ceil(P / tile rows) + E; where[sorted[i]] = i.  Counts and ranks in
// shared memory, one atomic a pair; a thread works on PLAN_RUN pairs at a time with their loads in
// flight together.  (Counting and sorting through atomics on global memory, the tiles listed by one
// thread: 16.1 us for 8,192 pairs, 6.9 for 256.)
#define PLAN_RUN 8
__global__ void __launch_bounds__(1024) moe_plan_kernel(const int* __restrict__ ids, int P, int E,
                                                        int num_tiles, int tile_rows, int* __restrict__ plan) {
    __shared__ int count[MOE_MAX_EXPERTS], start[MOE_MAX_EXPERTS];
    __shared__ int2 warp_total[32];
    int* offsets = plan + E;
    int* tile_expert = offsets + E + 1 + E;
    int* tile_row0 = tile_expert + num_tiles;
    int* sorted = tile_row0 + num_tiles;
    int* where = sorted + P;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid < E) count[tid] = 0;
    pdl_wait();
    pdl_launch_dependents();
    __syncthreads();
    for (int p0 = tid; p0 < P; p0 += PLAN_RUN * 1024) {
        int e[PLAN_RUN];
#pragma unroll
        for (int i = 0; i < PLAN_RUN; ++i) e[i] = p0 + i * 1024 < P ? ids[p0 + i * 1024] : -1;
#pragma unroll
        for (int i = 0; i < PLAN_RUN; ++i)
            if (e[i] >= 0 && e[i] < E) where[p0 + i * 1024] = atomicAdd(&count[e[i]], 1);
    }
    __syncthreads();
    // rows and tiles before every expert (thread = expert)
    const int n = tid < E ? count[tid] : 0, tiles = (n + tile_rows - 1) / tile_rows;
    int rows_upto = n, tiles_upto = tiles;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int a = __shfl_up_sync(0xffffffffu, rows_upto, o), b = __shfl_up_sync(0xffffffffu, tiles_upto, o);
        if (lane >= o) {
            rows_upto += a;
            tiles_upto += b;
        }
    }
    if (lane == 31) warp_total[warp] = make_int2(rows_upto, tiles_upto);
    __syncthreads();
    int all_tiles = 0, all_rows = 0;
    for (int i = 0; i < 32; ++i) {
        if (i < warp) {
            rows_upto += warp_total[i].x;
            tiles_upto += warp_total[i].y;
        }
        all_tiles += warp_total[i].y;
        all_rows += warp_total[i].x;
    }
    if (tid < E) {
        plan[tid] = n;
        start[tid] = offsets[tid] = rows_upto - n;
        if (tid == E - 1) offsets[E] = rows_upto;
        for (int i = 0; i < tiles; ++i) {
            tile_expert[tiles_upto - tiles + i] = tid;
            tile_row0[tiles_upto - tiles + i] = i * tile_rows;
        }
    }
    for (int i = all_tiles + tid; i < num_tiles; i += 1024) tile_expert[i] = -1;
    // (a pair whose id is no expert's is in no expert's rows; the list's end then names pair 0, so that whoever reads
    // the whole list, as the gather of rows does, stays in range)
    for (int i = all_rows + tid; i < P; i += 1024) sorted[i] = 0;
    __syncthreads();
    // (a product's result is written per pair, so the order within an expert changes no value)
    for (int p0 = tid; p0 < P; p0 += PLAN_RUN * 1024) {
        int e[PLAN_RUN], at[PLAN_RUN];
#pragma unroll
        for (int i = 0; i < PLAN_RUN; ++i) {
            const int p = p0 + i * 1024;
            e[i] = p < P ? ids[p] : -1;
            at[i] = p < P ? where[p] : 0;                  // (the thread's own rank)
        }
#pragma unroll
        for (int i = 0; i < PLAN_RUN; ++i) {
            const int p = p0 + i * 1024;
            if (p >= P) continue;
            const bool ok = e[i] >= 0 && e[i] < E;
            where[p] = ok ? start[e[i]] + at[i] : -1;
            if (ok) sorted[start[e[i]] + at[i]] = p;
        }
    }
}

// out[i] = x[sorted[i] / top]: the rows of every expert side by side; a warp a row, 16-byte pieces.
__global__ void __launch_bounds__(256) moe_gather_kernel(const bf16* __restrict__ x, int ldx,
                                                         const int* __restrict__ sorted, int top,
                                                         bf16* __restrict__ out, int ldo, int P, int row_pieces) {
    pdl_wait();
    pdl_launch_dependents();
    const int i = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (i >= P) return;
    const uint4* src = reinterpret_cast<const uint4*>(x + (size_t)(sorted[i] / top) * ldx);
    uint4* dst = reinterpret_cast<uint4*>(out + (size_t)i * ldo);
    for (int c = lane; c < row_pieces; c += 128) {
        uint4 v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (c + q * 32 < row_pieces) v[q] = src[c + q * 32];
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (c + q * 32 < row_pieces) dst[c + q * 32] = v[q];
    }
}

// ---------------------------------------------------------------- products
// MODE 0: gate|up with the activation: A rows are x[pair / top], W = w_gu[e] ([2 I, K]: I gate
// rows, then I up rows), C = act[pair][I].  MODE 1: down: A rows are act[pair], W = w_down[e]
// ([N, K = I]), C = y[pair][N] float32.
template <typename T, typename TC, int MODE>
__global__ void __launch_bounds__(256) moe_product_kernel(
    const T* __restrict__ A, int lda, const T* __restrict__ W, long long w_expert_stride, int ldw,
    TC* __restrict__ C, int ldc, const int* __restrict__ plan, int E, int num_tiles, int P, int top, int N, int K, int act, float limit, float alpha, const float* __restrict__ in_weights) {
    __shared__ __align__(16) float As[MOE_BK][MOE_BM + 4];
    __shared__ __align__(16) float Ws[MOE_BK][MOE_BN + 4];
    __shared__ __align__(16) float Us[MODE == 0 ? MOE_BK : 1][MOE_BN + 4];
    __shared__ int rows[MOE_BM];
    pdl_wait();
    const int* counts = plan;
    const int* offsets = plan + E;
    const int* tile_expert = offsets + E + 1 + E;
    const int* tile_row0 = tile_expert + num_tiles;
    const int* sorted = tile_row0 + num_tiles;
    const int e = tile_expert[blockIdx.y];
    if (e < 0) return;
    const int r0 = tile_row0[blockIdx.y];
    const int nrows = min(MOE_BM, counts[e] - r0);
    const int tid = threadIdx.x;
    if (tid < MOE_BM) rows[tid] = tid < nrows ? sorted[offsets[e] + r0 + tid] : -1;
    __syncthreads();
    const T* We = W + (size_t)e * w_expert_stride;
    const int ty = tid >> 4, tx = tid & 15;
    const int n0 = blockIdx.x * MOE_BN;
    float acc[4][4], acu[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = acu[i][j] = 0.f;
    for (int k0 = 0; k0 < K; k0 += MOE_BK) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int idx = tid + i * 256;
            const int row = idx >> 4, kk = idx & 15;
            const int gk = k0 + kk, gn = n0 + row;
            const int pr = rows[row];
            float av = 0.f;
            if (pr >= 0 && gk < K) av = to_float(A[(size_t)(MODE == 0 ? pr / top : pr) * lda + gk]);
            As[kk][row] = av;
            const bool in = gn < N && gk < K;
            Ws[kk][row] = in ? to_float(We[(size_t)gn * ldw + gk]) : 0.f;
            if (MODE == 0) Us[kk][row] = in ? to_float(We[(size_t)(N + gn) * ldw + gk]) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < MOE_BK; ++kk) {
            const float4 a = *reinterpret_cast<const float4*>(&As[kk][ty * 4]);
            const float4 b = *reinterpret_cast<const float4*>(&Ws[kk][tx * 4]);
            const float av[4] = {a.x, a.y, a.z, a.w};
            const float bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
            if (MODE == 0) {
                const float4 u = *reinterpret_cast<const float4*>(&Us[kk][tx * 4]);
                const float uv[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) acu[i][j] = fmaf(av[i], uv[j], acu[i][j]);
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int pr = rows[ty * 4 + i];
        if (pr < 0) continue;
        const float iw = MODE == 0 && in_weights != nullptr ? in_weights[pr] : 1.f;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int gn = n0 + tx * 4 + j;
            if (gn >= N) continue;
            float v = acc[i][j];
            if (MODE == 0) {
                // the gate and the up value are rounded to the activations' type first, as two
                // separate products would leave them
                const float gte = to_float(from_float<T>(v * iw)), up = to_float(from_float<T>(acu[i][j] * iw));
                v = act_mul_of(act, gte, up, limit, alpha);
            }
            C[(size_t)pr * ldc + gn] = from_float<TC>(v);
        }
    }
}

// ------------------------------------------------- products on tensor cores
// The same two products in bfloat16 on mma.sync (m16n8k16, float32 accumulation): a block owns up to
// 64 sorted rows of one expert and 64 output columns (MODE 0: 64 gate columns AND their 64 up
// columns, the activation in the epilogue), a warp 16 of the columns and all the rows, so that a
// fragment of the weights is read from shared memory once however many rows there are, and all four
// warps have work when an expert has a handful of rows.  A rows (gathered by the plan; only those
// that exist) and W rows arrive by 16-byte cp.async through a ring of STAGES k-blocks.  What bounds it at
// few rows is the weights' way from memory: the ring keeps (STAGES - 1) k-blocks of every resident
// block in flight.  Rows, K and the leading dimensions must be multiples of 8 elements.
#define MM_BN 64

template <int MODE, int BM, int BK> struct MoeStage {
    bf16 a[BM][BK + 8];
    bf16 w[MODE == 0 ? 2 : 1][MM_BN][BK + 8];
};

template <int MODE, int BM, int BK, int STAGES>
__global__ void __launch_bounds__(128) moe_product_mma_kernel(
    const bf16* __restrict__ A, int lda, const bf16* __restrict__ W, long long w_expert_stride, int ldw,
    void* __restrict__ Cv, int ldc, const int* __restrict__ plan, int E, int num_tiles, int top, int N,
    int K, int act, float limit, float alpha, const float* __restrict__ in_weights) {
    using namespace slb_mma;
    constexpr int NW = MODE == 0 ? 2 : 1, PIECES = BK / 8;
    extern __shared__ __align__(16) unsigned char mm_smem[];
    MoeStage<MODE, BM, BK>* ring = reinterpret_cast<MoeStage<MODE, BM, BK>*>(mm_smem);
    __shared__ int rows[BM];
    pdl_wait();
    const int* counts = plan;
    const int* offsets = plan + E;
    const int* tile_expert = offsets + E + 1 + E;
    const int* tile_row0 = tile_expert + num_tiles;
    const int* sorted = tile_row0 + num_tiles;
    const int e = tile_expert[blockIdx.y];
    if (e < 0) return;
    const int r0 = tile_row0[blockIdx.y];
    const int nrows = min(BM, counts[e] - r0);
    const int mtiles = (nrows + 15) >> 4;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid < BM) rows[tid] = tid < nrows ? sorted[offsets[e] + r0 + tid] : -1;
    __syncthreads();
    const bf16* We = W + (size_t)e * w_expert_stride;
    const int n0 = blockIdx.x * MM_BN;

    auto load = [&](int kb) {
        MoeStage<MODE, BM, BK>& st = ring[kb % STAGES];
        const int k0 = kb * BK;
#pragma unroll
        for (int idx = tid; idx < NW * MM_BN * PIECES; idx += 128) {
            const int r = idx / PIECES, c = (idx % PIECES) * 8, u = r / MM_BN, n = n0 + r % MM_BN;
            const bool ok = n < N && k0 + c < K;
            cp_async16(&st.w[u][r % MM_BN][c], We + (ok ? (size_t)(u * N + n) * ldw + k0 + c : 0), ok);
        }
        for (int idx = tid; idx < mtiles * 16 * PIECES; idx += 128) {
            const int r = idx / PIECES, c = (idx % PIECES) * 8, pr = rows[r];
            const bool ok = pr >= 0 && k0 + c < K;
            cp_async16(&st.a[r][c], A + (ok ? (size_t)(MODE == 0 ? pr / top : pr) * lda + k0 + c : 0), ok);
        }
    };

    float acc[NW][BM / 16][2][4];
#pragma unroll
    for (int u = 0; u < NW; ++u)
#pragma unroll
        for (int m = 0; m < BM / 16; ++m)
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int x = 0; x < 4; ++x) acc[u][m][j][x] = 0.f;

    const int nk = (K + BK - 1) / BK;
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) {
        if (s < nk) load(s);
        cp_async_commit();
    }
    for (int kb = 0; kb < nk; ++kb) {
        cp_async_wait<STAGES - 2>();
        __syncthreads();                                   // block kb is there; block kb - 1 has been read by all
        if (kb + STAGES - 1 < nk) load(kb + STAGES - 1);
        cp_async_commit();
        const MoeStage<MODE, BM, BK>& st = ring[kb % STAGES];
#pragma unroll
        for (int kk = 0; kk < BK / 16; ++kk) {
            unsigned b[NW][4];
#pragma unroll
            for (int u = 0; u < NW; ++u)
                ldmatrix_x4(b[u], &st.w[u][warp * 16 + (lane >> 4) * 8 + (lane & 7)][kk * 16 + ((lane >> 3) & 1) * 8]);
#pragma unroll
            for (int m = 0; m < BM / 16; ++m) {
                if (m >= mtiles) break;
                unsigned a[4];
                ldmatrix_x4(a, &st.a[m * 16 + (lane & 15)][kk * 16 + (lane >> 4) * 8]);
#pragma unroll
                for (int u = 0; u < NW; ++u) {
                    mma_bf16(acc[u][m][0], a, b[u][0], b[u][1]);
                    mma_bf16(acc[u][m][1], a, b[u][2], b[u][3]);
                }
            }
        }
    }
    const int tig = lane & 3;
#pragma unroll
    for (int m = 0; m < BM / 16; ++m) {
        if (m >= mtiles) break;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int pr = rows[m * 16 + (lane >> 2) + 8 * h];
            if (pr < 0) continue;
            const float iw = MODE == 0 && in_weights != nullptr ? in_weights[pr] : 1.f;
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int gn = n0 + warp * 16 + j * 8 + tig * 2;
                if (gn >= N) continue;                    // (N is even: both columns exist or neither)
                float v0 = acc[0][m][j][2 * h], v1 = acc[0][m][j][2 * h + 1];
                if (MODE == 0) {
                    auto rounded = [&](float x) { return __bfloat162float(__float2bfloat16_rn(x * iw)); };
                    v0 = act_mul_of(act, rounded(v0), rounded(acc[NW - 1][m][j][2 * h]), limit, alpha);
                    v1 = act_mul_of(act, rounded(v1), rounded(acc[NW - 1][m][j][2 * h + 1]), limit, alpha);
                    *reinterpret_cast<unsigned*>(reinterpret_cast<bf16*>(Cv) + (size_t)pr * ldc + gn) = pack_bf16(v0, v1);
                } else {
                    *reinterpret_cast<float2*>(reinterpret_cast<float*>(Cv) + (size_t)pr * ldc + gn) = make_float2(v0, v1);
                }
            }
        }
    }
}

// ----------------------------------------------------------------- combine
__device__ __forceinline__ void combine_load(const float* p, float (&v)[4]) {
    const float4 x = *reinterpret_cast<const float4*>(p);
    v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
}
__device__ __forceinline__ void combine_load(const bf16* p, float (&v)[4]) {
    const uint2 raw = *reinterpret_cast<const uint2*>(p);
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
    const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
__device__ __forceinline__ void combine_load(const bf16* p, float (&v)[8]) {
    const uint4 raw = *reinterpret_cast<const uint4*>(p);
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        v[2 * i] = __uint_as_float(w[i] << 16);
        v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
}
template <typename T> __device__ __forceinline__ void combine_load(const T* p, float (&v)[1]) { v[0] = to_float(p[0]); }
__device__ __forceinline__ void combine_store(float* p, const float (&v)[4]) {
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ void combine_store(bf16* p, const float (&v)[4]) {
    *reinterpret_cast<uint2*>(p) = make_uint2(slb_mma::pack_bf16(v[0], v[1]), slb_mma::pack_bf16(v[2], v[3]));
}
__device__ __forceinline__ void combine_store(bf16* p, const float (&v)[8]) {
    using slb_mma::pack_bf16;
    *reinterpret_cast<uint4*>(p) = make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
}
template <typename T> __device__ __forceinline__ void combine_store(T* p, const float (&v)[1]) { p[0] = from_float<T>(v[0]); }

// a thread V neighbouring columns; the experts' rows of four choices are in flight at once, the additions keep the
// order of the choice.  `where` (null: rows lie by pair): the row of every pair, -1: none.
template <typename T, typename TY, int V>
__global__ void __launch_bounds__(256) moe_combine_kernel(
    const TY* __restrict__ y, int ldy, const float* __restrict__ weights, const T* __restrict__ shared,
    int lds, T* __restrict__ out, int ldo, int top, int N, const int* __restrict__ where) {
    pdl_wait();
    pdl_launch_dependents();
    const int t = blockIdx.x;
    for (int c = (blockIdx.y * blockDim.x + threadIdx.x) * V; c < N; c += gridDim.y * blockDim.x * V) {
        float v[V];
#pragma unroll
        for (int e = 0; e < V; ++e) v[e] = 0.f;
        for (int k0 = 0; k0 < top; k0 += 4) {
            float r[4][V], w[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (k0 + k >= top) continue;
                const long long pair = (long long)t * top + k0 + k, row = where != nullptr ? where[pair] : pair;
#pragma unroll
                for (int e = 0; e < V; ++e) r[k][e] = 0.f;
                if (row >= 0) combine_load(y + (size_t)row * ldy + c, r[k]);
                w[k] = weights != nullptr ? weights[(size_t)t * top + k0 + k] : 1.f;
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (k0 + k >= top) continue;
#pragma unroll
                for (int e = 0; e < V; ++e) v[e] += w[k] * r[k][e];
            }
        }
        if (shared != nullptr) {
            float r[V];
            combine_load(shared + (size_t)t * lds + c, r);
#pragma unroll
            for (int e = 0; e < V; ++e) v[e] += r[e];
        }
        combine_store(out + (size_t)t * ldo + c, v);
    }
}

template <typename T, typename TY>
static int launch_moe_combine(const TY* y, int ldy, const float* weights, const T* shared, int lds, T* out, int ldo,
                              int T_, int top, int N, cudaStream_t st, const int* where = nullptr) {
    if (T_ <= 0) return 0;
    const uintptr_t half = (uintptr_t)shared | (uintptr_t)out;
    const bool vec = ((N | ldy | ldo | (shared != nullptr ? lds : 0)) & 3) == 0 && ((uintptr_t)y & (4 * sizeof(TY) - 1)) == 0 &&
                     (half & (4 * sizeof(T) - 1)) == 0;
    if constexpr (sizeof(TY) == 2 && sizeof(T) == 2) {
        // rows of a product in bfloat16, steps of many tokens: 16-byte pieces, a whole row in flight at once
        // (2,048 tokens of 4 rows of 2,048 anywhere in the list: 20.2 us with 8-byte pieces)
        if (((N | ldy | ldo | (shared != nullptr ? lds : 0)) & 7) == 0 && (((uintptr_t)y | half) & 15) == 0) {
            const int threads = N / 8 >= 256 ? 256 : (N / 8 + 31) / 32 * 32;
            return slb_launch(moe_combine_kernel<T, TY, 8>, dim3(T_), dim3(threads), 0, st, y, ldy, weights, shared, lds,
                              out, ldo, top, N, where);
        }
    }
    const int units = vec ? (N + 3) / 4 : N;
    const dim3 grid(T_, T_ < 256 ? (units + 255) / 256 : 1);
    if (vec)
        return slb_launch(moe_combine_kernel<T, TY, 4>, grid, dim3(256), 0, st, y, ldy, weights, shared, lds, out, ldo, top, N, where);
    return slb_launch(moe_combine_kernel<T, TY, 1>, grid, dim3(256), 0, st, y, ldy, weights, shared, lds, out, ldo, top, N, where);
}


template <typename T>
static int launch_moe_gate_up(const T* x, int ldx, const T* w_gu, int ldw, T* out, int lda,
                              const int* plan, int E, int P, int top, int I, int K, int act, float limit,
                              float alpha, const float* in_weights, cudaStream_t st) {
    if (P <= 0) return 0;
    if (E <= 0 || top <= 0 || I <= 0 || K <= 0 || act < 0 || act > 2 || (act == 2 && !(limit > 0.f))) return SLB_ERR_BAD_ARG;
    const int nt = moe_num_tiles(P, E, MOE_BM);
    if (nt > 65535) return SLB_ERR_TOO_LARGE;
    return slb_launch(moe_product_kernel<T, T, 0>, dim3((I + MOE_BN - 1) / MOE_BN, nt), dim3(256), 0, st, x,
                      ldx, w_gu, (long long)2 * I * ldw, ldw, out, lda, plan, E, nt, P, top, I, K, act, limit, alpha, in_weights);
}

template <typename T>
static int launch_moe_down(const T* act, int lda, const T* w_down, int ldw, float* y, int ldy,
                           const int* plan, int E, int P, int top, int N, int I, cudaStream_t st) {
    if (P <= 0) return 0;
    if (E <= 0 || top <= 0 || I <= 0 || N <= 0) return SLB_ERR_BAD_ARG;
    const int nt = moe_num_tiles(P, E, MOE_BM);
    if (nt > 65535) return SLB_ERR_TOO_LARGE;
    return slb_launch(moe_product_kernel<T, float, 1>, dim3((N + MOE_BN - 1) / MOE_BN, nt), dim3(256), 0, st,
                      act, lda, w_down, (long long)N * ldw, ldw, y, ldy, plan, E, nt, P, top, N, I, 0, 0.f, 0.f, (const float*)nullptr);
}

template <int MODE>
static int launch_moe_mma(const bf16* A, int lda, const bf16* W, long long stride, int ldw, void* C, int ldc,
                          const int* plan, int E, int P, int top, int N, int K, cudaStream_t st, int act = 0,
                          float limit = 0.f, float alpha = 0.f, const float* in_weights = nullptr) {
    if (P <= 0) return 0;
    if (E <= 0 || top <= 0 || N <= 0 || K <= 0 || K % 8 || lda % 8 || ldw % 8 || N % 2 || ldc % 2 ||
        ((uintptr_t)A & 15) || ((uintptr_t)W & 15) || (stride % 8) || act < 0 || act > 2 || (act == 2 && !(limit > 0.f)))
        return SLB_ERR_BAD_ARG;
    const int nt = moe_num_tiles(P, E);
    if (nt > 65535) return SLB_ERR_TOO_LARGE;
    const dim3 grid((N + MM_BN - 1) / MM_BN, nt);
#define MMF(BM, BK, ST)                                                                                               \
    do {                                                                                                              \
        static unsigned long long configured = 0;                                                                     \
        constexpr size_t smem = sizeof(MoeStage<MODE, BM, BK>) * ST;                                                  \
        const int rc = slb_configure(&configured, moe_product_mma_kernel<MODE, BM, BK, ST>, smem);                    \
        if (rc != 0) return rc;                                                                                       \
        return slb_launch(moe_product_mma_kernel<MODE, BM, BK, ST>, grid, dim3(128), smem, st, A, lda, W, stride, ldw, \
                          C, ldc, plan, E, nt, top, N, K, act, limit, alpha, in_weights);                             \
    } while (0)
    // Measured us, gate|up and down, 32 experts of 2,048 x 1,408 of 1 / 16 / 64 / 128 / 250 / 1,000 tokens, 4 experts
    // each: two stages of 32 with rows of warps and tiles of 64 rows 45.6 + 19.5 / 68.5 + 41.3 / 88.2 + 45.7 / 97.5 + 51.0
    // / 111 + 56 / 275 + 126; as below 20.2 + 13.5 / 57.0 + 32.5 / 70.1 + 38.1 / 86.9 + 49.5 / 114 + 53 / 244 + 129.  (At
    // 64 tokens 369 + 185 MB of weights: 56 + 28 us of the measured bandwidth.)  A third stage pays while few blocks
    // are resident, or while a block computes for long.
    const int rows = moe_tile_rows(P, E);
    if (rows == 16 && P <= E) MMF(16, 64, 3);
    if (rows == 16) MMF(16, 64, 2);
    if (rows == 32) MMF(32, 64, 3);
    MMF(64, 64, 2);
#undef MMF
}

extern "C" {
int slb_moe_gate_up_mma_bf16(const bf16* x, int ldx, const bf16* w_gu, int ldw, bf16* out, int lda,
                             const int* plan, int E, int P, int top, int I, int K, int act, float limit, float alpha,
                             const float* in_weights, cudaStream_t st) {
    return launch_moe_mma<0>(x, ldx, w_gu, (long long)2 * I * ldw, ldw, out, lda, plan, E, P, top, I, K, st, act, limit, alpha, in_weights);
}
int slb_moe_down_mma_bf16(const bf16* act, int lda, const bf16* w_down, int ldw, float* y, int ldy,
                          const int* plan, int E, int P, int top, int N, int I, cudaStream_t st) {
    return launch_moe_mma<1>(act, lda, w_down, (long long)N * ldw, ldw, y, ldy, plan, E, P, top, N, I, st);
}
int slb_moe_tile_rows(int P, int E) { return moe_tile_rows(P, E); }
static int launch_moe_route(const float* logits, int ldl, int T, int E, int groups, int keep, int top,
                            float route_scale, int renormalize, int score_fn, const float* correction,
                            int group_best, float norm_eps, int* ids, float* weights, cudaStream_t st) {
    if (T <= 0) return 0;
    if (E <= 0 || groups <= 0 || E % groups != 0 || keep <= 0 || keep > groups || top <= 0 ||
        top > (E / groups) * keep || score_fn < 0 || score_fn > 1 || group_best < 1)
        return SLB_ERR_BAD_ARG;
    if (E > MOE_MAX_EXPERTS || top > MOE_MAX_TOP) return SLB_ERR_TOO_LARGE;
    if (E <= MOE_FEW_EXPERTS && groups <= 32 && (groups == 1 || group_best == 1))
        return slb_launch(moe_route_few_kernel, dim3((T + 3) / 4), dim3(128), 0, st, logits, ldl, T, E, groups, keep, top,
                          route_scale, renormalize, score_fn, correction, norm_eps, ids, weights);
    const size_t smem = (size_t)4 * (2 * E + 2 * groups) * sizeof(float);
    return slb_launch(moe_route_kernel, dim3((T + 3) / 4), dim3(128), smem, st, logits, ldl, T, E, groups,
                      keep, top, route_scale, renormalize, score_fn, correction, group_best, norm_eps, ids,
                      weights);
}
// the softmax router whose groups score as their best expert
int slb_moe_route(const float* logits, int ldl, int T, int E, int groups, int keep, int top,
                  float route_scale, int renormalize, int* ids, float* weights, cudaStream_t st) {
    return launch_moe_route(logits, ldl, T, E, groups, keep, top, route_scale, renormalize, 0, nullptr, 1, 0.f,
                            ids, weights, st);
}
// every choice of the route kernel as an argument
int slb_moe_route_scored(const float* logits, int ldl, int T, int E, int groups, int keep, int top,
                         float route_scale, int renormalize, int score_fn, const float* correction,
                         int group_best, float norm_eps, int* ids, float* weights, cudaStream_t st) {
    return launch_moe_route(logits, ldl, T, E, groups, keep, top, route_scale, renormalize, score_fn, correction,
                            group_best, norm_eps, ids, weights, st);
}
int slb_router_logits_f32(const float* x, int ldx, const float* w, int ldw, float* logits, int ldl, int M,
                          int E, int K, cudaStream_t st) {
    if (M <= 0 || E <= 0) return 0;
    if (K <= 0) return SLB_ERR_BAD_ARG;
    return slb_launch(router_logits_kernel<float>, dim3((M + ROUTER_TOK - 1) / ROUTER_TOK, E), dim3(256), 0, st, x,
                      ldx, w, ldw, logits, ldl, M, E, K);
}
int slb_router_logits_bf16(const bf16* x, int ldx, const float* w, int ldw, float* logits, int ldl, int M,
                           int E, int K, cudaStream_t st) {
    if (M <= 0 || E <= 0) return 0;
    if (K <= 0) return SLB_ERR_BAD_ARG;
    return slb_launch(router_logits_kernel<bf16>, dim3((M + ROUTER_TOK - 1) / ROUTER_TOK, E), dim3(256), 0, st, x,
                      ldx, w, ldw, logits, ldl, M, E, K);
}
// float32 logits of a step of many tokens; 1: these sizes go elsewhere (rows of whole 16-byte pieces, K in
// chunks of RL_KC)
int slb_router_logits_tile_bf16(const bf16* x, int ldx, const float* w, int ldw, float* logits, int ldl, int M,
                                int E, int K, cudaStream_t st) {
    if (M <= 0 || E <= 0) return 0;
    if (K <= 0 || K % RL_KC || (ldx & 7) || (ldw & 3) || (((uintptr_t)x | (uintptr_t)w) & 15) || (E + RL_EXP - 1) / RL_EXP > 65535)
        return 1;
    constexpr size_t smem = sizeof(RouterStage) * RL_STAGES * 8;
    static_assert(smem >= 8 * RL_TOK * RL_EXP * sizeof(float), "the warps' sums fit into the rings");
    static unsigned long long configured = 0;
    const int rc = slb_configure(&configured, router_logits_tile_kernel, smem);
    if (rc != 0) return rc;
    return slb_launch(router_logits_tile_kernel, dim3((M + RL_TOK - 1) / RL_TOK, (E + RL_EXP - 1) / RL_EXP), dim3(256),
                      smem, st, x, ldx, w, ldw, logits, ldl, M, E, K);
}
static int launch_moe_plan(const int* ids, int P, int E, int rows, int* plan, cudaStream_t st) {
    if (P <= 0) return 0;
    if (E <= 0 || E > MOE_MAX_EXPERTS) return SLB_ERR_BAD_ARG;
    return slb_launch(moe_plan_kernel, dim3(1), dim3(1024), 0, st, ids, P, E, moe_num_tiles(P, E, rows), rows, plan);
}
// the plan of the products on tensor cores and of the library's ...
int slb_moe_plan_ints(int P, int E) { return moe_plan_ints(P, E, moe_tile_rows(P, E)); }
int slb_moe_plan(const int* ids, int P, int E, int* plan, cudaStream_t st) {
    return launch_moe_plan(ids, P, E, moe_tile_rows(P, E), plan, st);
}
// ... and of those on CUDA cores
int slb_moe_plan_simt_ints(int P, int E) { return moe_plan_ints(P, E, MOE_BM); }
int slb_moe_plan_simt(const int* ids, int P, int E, int* plan, cudaStream_t st) {
    return launch_moe_plan(ids, P, E, MOE_BM, plan, st);
}
int slb_moe_gate_up_f32(const float* x, int ldx, const float* w_gu, int ldw, float* out, int lda,
                        const int* plan, int E, int P, int top, int I, int K, int act, float limit, float alpha,
                        const float* in_weights, cudaStream_t st) {
    return launch_moe_gate_up<float>(x, ldx, w_gu, ldw, out, lda, plan, E, P, top, I, K, act, limit, alpha, in_weights, st);
}
int slb_moe_gate_up_bf16(const bf16* x, int ldx, const bf16* w_gu, int ldw, bf16* out, int lda,
                         const int* plan, int E, int P, int top, int I, int K, int act, float limit, float alpha,
                         const float* in_weights, cudaStream_t st) {
    return launch_moe_gate_up<bf16>(x, ldx, w_gu, ldw, out, lda, plan, E, P, top, I, K, act, limit, alpha, in_weights, st);
}
int slb_moe_down_f32(const float* act, int lda, const float* w_down, int ldw, float* y, int ldy,
                     const int* plan, int E, int P, int top, int N, int I, cudaStream_t st) {
    return launch_moe_down<float>(act, lda, w_down, ldw, y, ldy, plan, E, P, top, N, I, st);
}
int slb_moe_down_bf16(const bf16* act, int lda, const bf16* w_down, int ldw, float* y, int ldy,
                      const int* plan, int E, int P, int top, int N, int I, cudaStream_t st) {
    return launch_moe_down<bf16>(act, lda, w_down, ldw, y, ldy, plan, E, P, top, N, I, st);
}
int slb_moe_combine_f32(const float* y, int ldy, const float* weights, const float* shared, int lds,
                        float* out, int ldo, int T, int top, int N, cudaStream_t st) {
    return launch_moe_combine<float, float>(y, ldy, weights, shared, lds, out, ldo, T, top, N, st);
}
int slb_moe_combine_bf16(const float* y, int ldy, const float* weights, const bf16* shared, int lds,
                         bf16* out, int ldo, int T, int top, int N, cudaStream_t st) {
    return launch_moe_combine<bf16, float>(y, ldy, weights, shared, lds, out, ldo, T, top, N, st);
}
// the experts' rows in bfloat16, sorted by expert (as a product over sorted rows leaves them); the plan says where a
// pair's row is
int slb_moe_combine_bf16_sorted(const bf16* y, int ldy, const float* weights, const bf16* shared, int lds,
                                bf16* out, int ldo, const int* plan, int E, int T, int top, int N, cudaStream_t st) {
    if (E <= 0 || plan == nullptr) return SLB_ERR_BAD_ARG;
    const int P = T * top;
    return launch_moe_combine<bf16, bf16>(y, ldy, weights, shared, lds, out, ldo, T, top, N, st,
                                          plan + 3 * E + 1 + 2 * moe_num_tiles(P, E) + P);
}
// ... in float32
int slb_moe_combine_bf16_sorted_f32(const float* y, int ldy, const float* weights, const bf16* shared, int lds,
                                    bf16* out, int ldo, const int* plan, int E, int T, int top, int N, cudaStream_t st) {
    if (E <= 0 || plan == nullptr) return SLB_ERR_BAD_ARG;
    const int P = T * top;
    return launch_moe_combine<bf16, float>(y, ldy, weights, shared, lds, out, ldo, T, top, N, st,
                                           plan + 3 * E + 1 + 2 * moe_num_tiles(P, E) + P);
}
// out[i] = the input row of the i-th pair of the plan's list; rows of whole 16-byte pieces
int slb_moe_gather_bf16(const bf16* x, int ldx, const int* plan, int E, int P, int top, int K, bf16* out, int ldo,
                        cudaStream_t st) {
    if (P <= 0) return 0;
    if (E <= 0 || top <= 0 || K <= 0 || ((K | ldx | ldo) & 7) || (((uintptr_t)x | (uintptr_t)out) & 15))
        return SLB_ERR_BAD_ARG;
    return slb_launch(moe_gather_kernel, dim3((P + 7) / 8), dim3(256), 0, st, x, ldx,
                      plan + 3 * E + 1 + 2 * moe_num_tiles(P, E), top, out, ldo, P, K / 8);
}
}

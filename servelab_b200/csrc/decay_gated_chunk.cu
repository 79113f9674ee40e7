// Linear attention with a decay of its own for every token and key channel, for portions of
// prompts: the recurrence
//
//     S_t = diag(alpha_t) S_{t-1} + k_t v_t^T,   o_t = S_t^T q_t
//
// cut into chunks of 32 tokens.  With l_t = log alpha_t and L_t = l_first + ... + l_t inside a chunk
// (per key channel d), and S the state that enters the chunk,
//
//     o_t   = sum_d q_t[d] e^(L_t[d]) S[d][:]  +  sum_{j <= t} A[t][j] v_j,
//     A[t][j] = sum_d q_t[d] k_j[d] e^(L_t[d] - L_j[d]),
//     S_out = diag(e^(L_last)) S + sum_j diag(e^(L_last - L_j)) k_j v_j^T.
//
// With a bonus the result reads the state before the token's own update and the token itself through a
// learned factor per key channel, o_t = (S_{t-1} + diag(bonus) k_t v_t^T)^T q_t: then e^(L_{t-1}[d])
// takes the place of e^(L_t[d]) in o_t and in A[t][j] for j < t, and A[t][t] = sum_d q_t bonus k_t.
//
// Every exponent is a difference L_t - L_j with j <= t, or L_t itself: never positive, so nothing
// overflows however fast a channel decays (a factorised form q e^L . k e^-L would).  All
// arithmetic is float32 on the CUDA cores: the logarithms of the decays, their sums, the
// exponentials, the products and the state (what enters a recurrence stays 32-bit also where the
// projections are bfloat16).
//
// Two launches, or four:
//   1. `prep` per (chunk, head): L for the chunk's tokens and the masked scores A; a record in a work
//      buffer holds the queries times e^(L_t), the keys times e^(L_last - L_j), A and e^(L_last),
//      padded as the second launch wants them in shared memory;
//   2. `walk` per (request, head, slice of EV value columns): the chunks in order with the slice of the
//      state in shared memory, the next chunk's record fetched by one bulk copy while this one is
//      worked on; outputs and the new state from the same rows.
//      The state of a chunk never goes to memory;
//   or, for long requests of few heads and values, whose walk would be a long chain on few SMs:
//   2. `local` per (chunk, head, 64 value columns): the sum that a chunk adds to the state, into a second buffer;
//   3. `scan` per (request, head, state element): the buffer is left holding the state that ENTERS every chunk;
//   4. `out` per (chunk, head, 64 value columns): the outputs.
//      The states are written and read twice (67 MB each way for 2,048 tokens of 8 heads of 128 x 256), but no
//      chunk waits for another outside the scan.
// The result differs from the token-by-token kernel by float32 rounding only, and so does
// the result of a prompt cut elsewhere.
#include "decay_attention.cuh"
#include "mma_util.cuh"

#define GC_CHUNK 32
#define GC_LA 36                             // row stride of A
#define GC_MAX_D 256

// 0, or 1: the wait for a chunk's record gave up and the request's rows of that launch are not written
SLB_DEFINE_STATUS_WORD(gated_chunk_status_word, slb_decay_gated_chunk_status)

struct GatedChunkArgs {
    DecayAttnArgs a;
    const int* tile_seq; const int* tile_row0; int num_tiles;
    float* work;                             // [num_tiles][H][gc_floats(D)]
    float* states;                           // [num_tiles][H][D][Dv] for the form without a walk; null: the walk
};

// A record: q~ and k~ [32][Dp + 4] (zero rows beyond the chunk's tokens, zero columns beyond D), A [32][36],
// e^(L_last) [Dp].  With 4 floats of padding eight neighbouring rows read 16 bytes each from 32 banks.
__host__ __device__ constexpr int gc_pad(int D) { return (D + 7) & ~7; }
__host__ __device__ constexpr int gc_ld(int D) { return gc_pad(D) + 4; }
__host__ __device__ constexpr int gc_floats(int D) {
    return 2 * GC_CHUNK * gc_ld(D) + GC_CHUNK * GC_LA + gc_pad(D);
}

__device__ __forceinline__ bool gc_tile(const GatedChunkArgs& c, int tile, int& t0, int& n) {
    const DecayAttnArgs& a = c.a;
    const int s = c.tile_seq[tile];
    const int q0 = a.cu_q[s];
    const int row0 = c.tile_row0[tile];
    n = min(GC_CHUNK, a.cu_q[s + 1] - q0 - row0);
    t0 = q0 + row0;
    return n > 0;
}

// ------------------------------------------------------------------ 1. logarithms and scores
// The scores: thread (ti, tj, quarter of the channels) sums the pairs (ti + 8 i, tj + 8 jj), i >= jj, so that
// 16 loads of 16 bytes serve 10 pairs of 4 channels (a pair a thread read four floats for every
// channel: 46 us for 2,048 tokens of 8 heads of 128, most of it those loads).
#define GC_PAIRS 10
template <typename T>
__global__ void __launch_bounds__(256) gated_chunk_prep_kernel(const GatedChunkArgs c) {
    extern __shared__ __align__(16) float gc_smem[];
    pdl_wait();
    pdl_launch_dependents();
    const DecayAttnArgs& a = c.a;
    const int tile = blockIdx.x, h = blockIdx.y;
    int t0, n;
    if (!gc_tile(c, tile, t0, n)) return;
    const int D = a.D, Dp = gc_pad(D), LD = gc_ld(D);
    float* Ls = gc_smem;                         // [GC_CHUNK][LD]
    float* qs = Ls + GC_CHUNK * LD;
    float* ks = qs + GC_CHUNK * LD;
    float* rec = c.work + ((size_t)tile * a.H + h) * gc_floats(D);
    float* gq = rec, *gk = gq + GC_CHUNK * LD, *gA = gk + GC_CHUNK * LD, *gG = gA + GC_CHUNK * GC_LA;
    const T* proj = reinterpret_cast<const T*>(a.proj);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // the logarithms of the decays, every (token, channel) on a thread of its own ...
    for (int d = lane; d < Dp; d += 32) {                  // (a warp has the four tokens from 4 warp)
        const bool live = d < D;
        const float bias = live && a.gate_bias != nullptr ? a.gate_bias[h * D + d] : 0.f;
        float z[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int j = warp * 4 + i;
            z[i] = live && j < n ? a.gate_z[(size_t)(t0 + j) * a.ld_gate + h * D + d] + bias : 0.f;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
            Ls[(warp * 4 + i) * LD + d] = live && warp * 4 + i < n ? da_log_decay(z[i], a.gate_kind, a.gate_inv_tau) : 0.f;
    }
    __syncthreads();
    // ... then their running sums, a channel a thread, in the order of the tokens (beyond them the sum stays)
    for (int d = threadIdx.x; d < Dp; d += blockDim.x) {
        float l[GC_CHUNK], run = 0.f;
#pragma unroll
        for (int j = 0; j < GC_CHUNK; ++j) l[j] = Ls[j * LD + d];
#pragma unroll
        for (int j = 0; j < GC_CHUNK; ++j) Ls[j * LD + d] = run += l[j];
        gG[d] = decay_exp(run);
    }
    __syncthreads();
    const bool plain = a.act == 0 && a.rot_dims == 0;      // (then a token's loads can all be in flight at once)
    for (int d = lane; d < Dp; d += 32) {
        const float last = Ls[(GC_CHUNK - 1) * LD + d];
        const T* at = proj + (size_t)(t0 + warp * 4) * a.ld + h * D + d;
        float qv[4], kv[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int j = warp * 4 + i;
            qv[i] = kv[i] = 0.f;
            if (j < n && d < D) {
                if (plain) {
                    qv[i] = to_float(at[(size_t)i * a.ld + a.q_off]);
                    kv[i] = to_float(at[(size_t)i * a.ld + a.k_off]);
                } else {
                    const int pos = a.positions[t0 + j];
                    qv[i] = da_prepared(at + (size_t)i * a.ld + a.q_off - d, d, pos, a);
                    kv[i] = da_prepared(at + (size_t)i * a.ld + a.k_off - d, d, pos, a);
                }
            }
        }
        float before = warp > 0 ? Ls[(warp * 4 - 1) * LD + d] : 0.f;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int j = warp * 4 + i;
            const float L = Ls[j * LD + d], q = qv[i] * a.q_scale, k = kv[i] * a.k_scale;
            qs[j * LD + d] = q;
            ks[j * LD + d] = k;
            gq[j * LD + d] = q * expf(a.bonus == nullptr ? L : before);
            gk[j * LD + d] = k * expf(last - L);
            before = L;
        }
    }
    __syncthreads();
    const int tj = threadIdx.x & 7, ti = (threadIdx.x >> 3) & 7, part = threadIdx.x >> 6;
    float acc[GC_PAIRS];
#pragma unroll
    for (int p = 0; p < GC_PAIRS; ++p) acc[p] = 0.f;
    const int back = a.bonus == nullptr ? 0 : 1;           // (a bonus reads the state before the token's own update)
    const float* bonus = a.bonus == nullptr ? nullptr : a.bonus + h * D;
    for (int d = part * 4; d < Dp; d += 16) {
        float4 q[4], k[4], lt[4], lj[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int t = ti + 8 * i, j = tj + 8 * i;
            q[i] = *reinterpret_cast<const float4*>(qs + t * LD + d);
            lt[i] = *reinterpret_cast<const float4*>(Ls + max(t - back, 0) * LD + d);
            k[i] = *reinterpret_cast<const float4*>(ks + j * LD + d);
            lj[i] = *reinterpret_cast<const float4*>(Ls + j * LD + d);
        }
        // (the exponent is <= 0 where the pair counts; the one-instruction 2^x is exact to 2 ulp there, and its
        // argument's rounding weighs on terms that are small by the same factor)
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int jj = 0; jj <= i; ++jj) {
                float x0 = lt[i].x - lj[jj].x, x1 = lt[i].y - lj[jj].y, x2 = lt[i].z - lj[jj].z, x3 = lt[i].w - lj[jj].w;
                if (i == jj) {                             // (pairs above the diagonal are summed and not used)
                    x0 = fminf(x0, 0.f);
                    x1 = fminf(x1, 0.f);
                    x2 = fminf(x2, 0.f);
                    x3 = fminf(x3, 0.f);
                }
                float e0 = __expf(x0), e1 = __expf(x1), e2 = __expf(x2), e3 = __expf(x3);
                if (i == jj && bonus != nullptr && ti == tj) {
                    e0 = d < D ? bonus[d] : 0.f;
                    e1 = d + 1 < D ? bonus[d + 1] : 0.f;
                    e2 = d + 2 < D ? bonus[d + 2] : 0.f;
                    e3 = d + 3 < D ? bonus[d + 3] : 0.f;
                }
                float& v = acc[i * (i + 1) / 2 + jj];
                v = fmaf(q[i].x * k[jj].x, e0, v);
                v = fmaf(q[i].y * k[jj].y, e1, v);
                v = fmaf(q[i].z * k[jj].z, e2, v);
                v = fmaf(q[i].w * k[jj].w, e3, v);
            }
    }
    __syncthreads();
    float* sums = qs;                                      // [4][GC_PAIRS][64] (the queries have been read)
#pragma unroll
    for (int p = 0; p < GC_PAIRS; ++p) sums[(part * GC_PAIRS + p) * 64 + ti * 8 + tj] = acc[p];
    __syncthreads();
    for (int e = threadIdx.x; e < GC_CHUNK * GC_CHUNK; e += blockDim.x) {
        const int t = e / GC_CHUNK, j = e % GC_CHUNK, i = t >> 3, jj = j >> 3;
        float v = 0.f;
        if (j <= t && t < n) {
            const float* s = sums + (i * (i + 1) / 2 + jj) * 64 + (t & 7) * 8 + (j & 7);
            v = (s[0] + s[GC_PAIRS * 64]) + (s[2 * GC_PAIRS * 64] + s[3 * GC_PAIRS * 64]);
        }
        gA[t * GC_LA + j] = v;
    }
}

// ------------------------------------------------------------------ 2. the walk over the chunks
// Half of the warps form the outputs: a warp has every eighth group of four channels (and of four tokens j), a
// lane 4 tokens by EV / 4 columns, and the warps' parts are added through shared memory.  The other half
// forms the state that leaves the chunk in a second buffer, a thread 4 rows by 2 columns at a time.  Both
// read 16 bytes of a row at a time; 32 (2 D + 32) EV FFMA a chunk bound it, with the latency of shared memory
// behind them.  2,048 tokens of 8 heads of 128 x 256: 123 us, where the chunks' sums, the scan and the outputs
// took 171 and the scores 46 instead of 36.  DP: the padded head size (0: any).
template <typename T, int EV, int DP>
__global__ void __launch_bounds__(512, 1) gated_chunk_walk_kernel(const GatedChunkArgs c) {
    extern __shared__ __align__(16) float gc_smem[];
    constexpr int CV = EV / 4, E2 = EV / 2, DG = 256 / E2;
    __shared__ int first_s;
    __shared__ __align__(8) uint64_t bars[2];
    pdl_wait();
    const DecayAttnArgs& a = c.a;
    const int s = blockIdx.x, h = blockIdx.y, e0 = blockIdx.z * EV;
    const int q0 = a.cu_q[s];
    const int qlen = a.cu_q[s + 1] - q0;
    if (qlen <= 0) return;
    const int slot = a.state_slots[s];
    if (slot < 0 || slot >= a.num_slots) return;
    const int tid = threadIdx.x;
    if (tid == 0) {
        first_s = c.num_tiles;
        for (int i = 0; i < 2; ++i) slb_mma::mbar_init(&bars[i], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    for (int i = tid; i < c.num_tiles; i += 512)     // a request's chunks are neighbours in the list, in order
        if (c.tile_seq[i] == s) { atomicMin(&first_s, i); break; }
    __syncthreads();
    const int first = first_s;
    const int count = (qlen + GC_CHUNK - 1) / GC_CHUNK;
    if (first + count > c.num_tiles) return;
    const int D = a.D, Dv = a.Dv, Dp = DP ? DP : gc_pad(D), LD = Dp + 4;
    const int rec_floats = 2 * GC_CHUNK * LD + GC_CHUNK * GC_LA + Dp;
    float* stages = gc_smem;
    float* Ss = stages + 2 * rec_floats;             // [2][Dp][EV]: the state's columns entering even and odd chunks
    float* Vs = Ss + 2 * Dp * EV;                    // [2][32][EV]
    float* red = Vs + 2 * GC_CHUNK * EV;             // [8][32][EV]
    const float* recs = c.work + ((size_t)first * a.H + h) * rec_floats;
    auto fetch = [&](int k) {
        slb_mma::mbar_arrive_expect_tx(&bars[k & 1], (uint32_t)rec_floats * 4);
        slb_mma::bulk_copy_g2s(stages + (k & 1) * rec_floats, recs + (size_t)k * a.H * rec_floats,
                               (uint32_t)rec_floats * 4, &bars[k & 1]);
    };
    if (tid == 0) fetch(0);
    float* gS = a.state + (size_t)slot * (size_t)a.state_stride + (size_t)h * D * Dv;
    for (int idx = tid; idx < Dp * EV; idx += 512) {
        const int d = idx / EV, e = idx % EV;
        Ss[idx] = d < D && e0 + e < Dv ? gS[(size_t)d * Dv + e0 + e] : 0.f;
    }
    // the values of a chunk: a (token, column) pair a thread, as it lies in memory until it is stored
    const int ve = tid % EV, vj = tid / EV;
    const bool v_mine = tid < GC_CHUNK * EV && e0 + ve < Dv;
    const T* vp = reinterpret_cast<const T*>(a.proj) + (size_t)(q0 + vj) * a.ld + a.v_off + h * Dv + e0 + ve;
    T v_next = from_float<T>(0.f);
    auto load_v = [&](int k) {
        if (v_mine && k * GC_CHUNK + vj < qlen) v_next = vp[(size_t)k * GC_CHUNK * a.ld];
        else v_next = from_float<T>(0.f);
    };
    auto store_v = [&](int k) {
        float v = to_float(v_next);
        if (a.act == 1) v = da_silu(v);
        if (tid < GC_CHUNK * EV) Vs[((k & 1) * GC_CHUNK + vj) * EV + ve] = v;
    };
    load_v(0);
    store_v(0);
    const int warp = (tid >> 5) & 7, lane = tid & 31, ty = lane >> 2, tx = lane & 3, half = tid & 255;
    const bool outputs = tid < 256;
    const bool wide = (Dv & 3) == 0 && (a.ldo & 3) == 0 && ((uintptr_t)a.out & 15) == 0;
    for (int k = 0; k < count; ++k) {
        const bool there = slb_mma::mbar_wait(&bars[k & 1], (k >> 1) & 1);
        if (!__syncthreads_and(there)) {             // the copy did not come in time: say so, and give it its limit once
            if (tid == 0) {                          // more before the block's shared memory goes to another
                atomicCAS(&gated_chunk_status_word, 0, 1);
                slb_mma::mbar_wait(&bars[k & 1], (k >> 1) & 1);
            }
            return;
        }
        const bool more = k + 1 < count;
        if (more && tid == 256) fetch(k + 1);
        if (more) load_v(k + 1);
        const float* qd = stages + (k & 1) * rec_floats, *kd = qd + GC_CHUNK * LD, *A = kd + GC_CHUNK * LD;
        const float* G = A + GC_CHUNK * GC_LA, *V = Vs + (k & 1) * GC_CHUNK * EV;
        const float* S = Ss + (k & 1) * Dp * EV;
        if (outputs) {
            float acc[4][CV];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int x = 0; x < CV; ++x) acc[i][x] = 0.f;
            // four rows of the right operand against a 16-byte piece of four rows of the left one
            auto piece = [&](const float* left, int ld, const float* right) {
                float4 l[4];
                float r[4][CV];
#pragma unroll
                for (int i = 0; i < 4; ++i) l[i] = *reinterpret_cast<const float4*>(left + (ty + 8 * i) * ld);
#pragma unroll
                for (int y = 0; y < 4; ++y) {
                    if constexpr (CV == 4) {
                        const float4 v = *reinterpret_cast<const float4*>(right + y * EV + tx * CV);
                        r[y][0] = v.x; r[y][1] = v.y; r[y][2] = v.z; r[y][3] = v.w;
                    } else {
                        const float2 v = *reinterpret_cast<const float2*>(right + y * EV + tx * CV);
                        r[y][0] = v.x; r[y][1] = v.y;
                    }
                }
#pragma unroll
                for (int y = 0; y < 4; ++y)
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float lv = y == 0 ? l[i].x : y == 1 ? l[i].y : y == 2 ? l[i].z : l[i].w;
#pragma unroll
                        for (int x = 0; x < CV; ++x) acc[i][x] = fmaf(lv, r[y][x], acc[i][x]);
                    }
            };
            if constexpr (DP != 0) {
#pragma unroll
                for (int g = 0; g < DP / 32; ++g) piece(qd + warp * 4 + g * 32, LD, S + (warp * 4 + g * 32) * EV);
            } else {
                for (int d = warp * 4; d < Dp; d += 32) piece(qd + d, LD, S + d * EV);
            }
            piece(A + warp * 4, GC_LA, V + warp * 4 * EV);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float* p = red + (warp * GC_CHUNK + ty + 8 * i) * EV + tx * CV;
                if constexpr (CV == 4) *reinterpret_cast<float4*>(p) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
                else *reinterpret_cast<float2*>(p) = make_float2(acc[i][0], acc[i][1]);
            }
            asm volatile("bar.sync 1, 256;" ::: "memory");
            if (half < GC_CHUNK * EV / 4) {
                const int t = k * GC_CHUNK + half / (EV / 4), e = e0 + (half % (EV / 4)) * 4;
                float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (int w = 0; w < 8; ++w) {
                    const float4 p = *reinterpret_cast<const float4*>(red + w * GC_CHUNK * EV + half * 4);
                    o.x += p.x; o.y += p.y; o.z += p.z; o.w += p.w;
                }
                if (t < qlen && e < Dv) {
                    float* dst = a.out + (size_t)(q0 + t) * a.ldo + h * Dv + e;
                    if (wide) {
                        *reinterpret_cast<float4*>(dst) = o;
                    } else {
                        dst[0] = o.x;
                        if (e + 1 < Dv) dst[1] = o.y;
                        if (e + 2 < Dv) dst[2] = o.z;
                        if (e + 3 < Dv) dst[3] = o.w;
                    }
                }
            }
        } else {
            float* S2 = Ss + ((k + 1) & 1) * Dp * EV;
            const int e2 = (half % E2) * 2;
            for (int d = half / E2 * 4; d < Dp; d += DG * 4) {
                float u[4][2];
#pragma unroll
                for (int i = 0; i < 4; ++i) u[i][0] = u[i][1] = 0.f;
#pragma unroll 16
                for (int j = 0; j < GC_CHUNK; ++j) {
                    const float4 kv = *reinterpret_cast<const float4*>(kd + j * LD + d);
                    const float2 v = *reinterpret_cast<const float2*>(V + j * EV + e2);
                    u[0][0] = fmaf(kv.x, v.x, u[0][0]); u[0][1] = fmaf(kv.x, v.y, u[0][1]);
                    u[1][0] = fmaf(kv.y, v.x, u[1][0]); u[1][1] = fmaf(kv.y, v.y, u[1][1]);
                    u[2][0] = fmaf(kv.z, v.x, u[2][0]); u[2][1] = fmaf(kv.z, v.y, u[2][1]);
                    u[3][0] = fmaf(kv.w, v.x, u[3][0]); u[3][1] = fmaf(kv.w, v.y, u[3][1]);
                }
                const float4 g = *reinterpret_cast<const float4*>(G + d);
                const float gg[4] = {g.x, g.y, g.z, g.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float2 st = *reinterpret_cast<const float2*>(S + (d + i) * EV + e2);
                    *reinterpret_cast<float2*>(S2 + (d + i) * EV + e2) =
                        make_float2(fmaf(gg[i], st.x, u[i][0]), fmaf(gg[i], st.y, u[i][1]));
                }
            }
        }
        if (more) store_v(k + 1);
    }
    __syncthreads();
    pdl_launch_dependents();
    const float* S = Ss + (count & 1) * Dp * EV;
    for (int idx = tid; idx < D * EV; idx += 512) {
        const int d = idx / EV, e = idx % EV;
        if (e0 + e < Dv) gS[(size_t)d * Dv + e0 + e] = S[idx];
    }
}

// ------------------------------------------------------------------ 2b. what a chunk adds to the state
// Thread (dy, ex): state rows dy, dy + 16, ... and value columns 4 ex .. 4 ex + 3 of the slice.
#define GC_EV 64
template <typename T>
__device__ __forceinline__ void gc_stage_values(const GatedChunkArgs& c, int h, int e0, int t0, int n, float* vs) {
    const DecayAttnArgs& a = c.a;
    const T* v = reinterpret_cast<const T*>(a.proj) + (size_t)t0 * a.ld + a.v_off + h * a.Dv + e0;
#pragma unroll
    for (int i = 0; i < GC_CHUNK * GC_EV / 256; ++i) {
        const int j = (threadIdx.x >> 6) + 4 * i, e = threadIdx.x & 63;
        float x = 0.f;
        if (j < n && e0 + e < a.Dv) x = to_float(v[(size_t)j * a.ld + e]);
        vs[j * GC_EV + e] = a.act == 1 ? da_silu(x) : x;
    }
}
template <typename T, int R>
__global__ void __launch_bounds__(256) gated_chunk_local_kernel(const GatedChunkArgs c) {
    extern __shared__ __align__(16) float gc_smem[];
    pdl_wait();
    pdl_launch_dependents();
    const DecayAttnArgs& a = c.a;
    const int tile = blockIdx.x, h = blockIdx.y, e0 = blockIdx.z * GC_EV;
    int t0, n;
    if (!gc_tile(c, tile, t0, n)) return;
    const int D = a.D, Dv = a.Dv, LD = gc_ld(D);
    float* kk = gc_smem;                         // [32][LD]: the record's keys
    float* vs = kk + GC_CHUNK * LD;              // [32][GC_EV]
    const float* rec = c.work + ((size_t)tile * a.H + h) * gc_floats(D) + GC_CHUNK * LD;
    for (int i = threadIdx.x * 4; i < GC_CHUNK * LD; i += 1024)
        *reinterpret_cast<float4*>(kk + i) = *reinterpret_cast<const float4*>(rec + i);
    gc_stage_values<T>(c, h, e0, t0, n, vs);
    __syncthreads();
    const int ex = threadIdx.x & 15, dy = threadIdx.x >> 4;
    float acc[R][4];
#pragma unroll
    for (int i = 0; i < R; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
    for (int j = 0; j < n; ++j) {
        const float4 v = *reinterpret_cast<const float4*>(vs + j * GC_EV + ex * 4);
        const float* kj = kk + j * LD + dy;
#pragma unroll
        for (int i = 0; i < R; ++i) {
            if (dy + 16 * i >= D) break;
            const float k = kj[16 * i];
            acc[i][0] = fmaf(k, v.x, acc[i][0]); acc[i][1] = fmaf(k, v.y, acc[i][1]);
            acc[i][2] = fmaf(k, v.z, acc[i][2]); acc[i][3] = fmaf(k, v.w, acc[i][3]);
        }
    }
    float* w = c.states + ((size_t)tile * a.H + h) * (size_t)D * Dv + e0 + ex * 4;
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const int d = dy + 16 * i;
        if (d >= D) break;
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (e0 + ex * 4 + u < Dv) w[(size_t)d * Dv + u] = acc[i][u];
    }
}

// ------------------------------------------------------------------ 3b. the states that enter the chunks
#define GC_SCAN_BATCH 16
__global__ void __launch_bounds__(256) gated_chunk_scan_kernel(const GatedChunkArgs c) {
    __shared__ int first_s;
    pdl_wait();
    pdl_launch_dependents();
    const DecayAttnArgs& a = c.a;
    const int s = blockIdx.x, h = blockIdx.y;
    const int qlen = a.cu_q[s + 1] - a.cu_q[s];
    if (qlen <= 0) return;
    const int slot = a.state_slots[s];
    if (slot < 0 || slot >= a.num_slots) return;
    if (threadIdx.x == 0) first_s = c.num_tiles;
    __syncthreads();
    for (int i = threadIdx.x; i < c.num_tiles; i += 256)       // (a request's chunks are neighbours, in order)
        if (c.tile_seq[i] == s) { atomicMin(&first_s, i); break; }
    __syncthreads();
    const int elems = a.D * a.Dv, idx = blockIdx.z * 256 + threadIdx.x;
    const int first = first_s, count = (qlen + GC_CHUNK - 1) / GC_CHUNK;
    if (idx >= elems || first + count > c.num_tiles) return;
    const int rec = gc_floats(a.D);
    float* sp = a.state + (size_t)slot * (size_t)a.state_stride + (size_t)h * elems + idx;
    float* wp = c.states + ((size_t)first * a.H + h) * (size_t)elems + idx;
    const float* gp = c.work + ((size_t)first * a.H + h) * rec + rec - gc_pad(a.D) + idx / a.Dv;
    const size_t step = (size_t)a.H * elems, gstep = (size_t)a.H * rec;
    float S = *sp;
    for (int k0 = 0; k0 < count; k0 += GC_SCAN_BATCH) {
        float add[GC_SCAN_BATCH], g[GC_SCAN_BATCH];
#pragma unroll
        for (int u = 0; u < GC_SCAN_BATCH; ++u) {
            add[u] = k0 + u < count ? wp[u * step] : 0.f;
            g[u] = k0 + u < count ? gp[u * gstep] : 1.f;
        }
#pragma unroll
        for (int u = 0; u < GC_SCAN_BATCH; ++u)
            if (k0 + u < count) {
                wp[u * step] = S;
                S = fmaf(g[u], S, add[u]);
            }
        wp += GC_SCAN_BATCH * step;
        gp += GC_SCAN_BATCH * gstep;
    }
    *sp = S;
}

// ------------------------------------------------------------------ 4b. the chunk's outputs
// Thread (ty, ex): tokens ty and ty + 16 of the chunk, value columns 4 ex .. 4 ex + 3 of the slice.
template <typename T>
__global__ void __launch_bounds__(256) gated_chunk_out_kernel(const GatedChunkArgs c) {
    extern __shared__ __align__(16) float gc_smem[];
    pdl_wait();
    pdl_launch_dependents();
    const DecayAttnArgs& a = c.a;
    const int tile = blockIdx.x, h = blockIdx.y, e0 = blockIdx.z * GC_EV;
    int t0, n;
    if (!gc_tile(c, tile, t0, n)) return;
    const int slot = a.state_slots[c.tile_seq[tile]];
    if (slot < 0 || slot >= a.num_slots) return;
    const int D = a.D, Dv = a.Dv, Dp = gc_pad(D), LD = gc_ld(D);
    float* q = gc_smem;                          // [32][LD]: the record's queries
    float* A = q + GC_CHUNK * LD;                // [32][GC_LA]
    float* vs = A + GC_CHUNK * GC_LA;            // [32][GC_EV]
    float* S = vs + GC_CHUNK * GC_EV;            // [Dp][GC_EV]: the entering state's slice, zeros beyond it
    const float* rec = c.work + ((size_t)tile * a.H + h) * gc_floats(D);
    for (int i = threadIdx.x * 4; i < GC_CHUNK * LD; i += 1024)
        *reinterpret_cast<float4*>(q + i) = *reinterpret_cast<const float4*>(rec + i);
    for (int i = threadIdx.x * 4; i < GC_CHUNK * GC_LA; i += 1024)
        *reinterpret_cast<float4*>(A + i) = *reinterpret_cast<const float4*>(rec + 2 * GC_CHUNK * LD + i);
    gc_stage_values<T>(c, h, e0, t0, n, vs);
    const float* w = c.states + ((size_t)tile * a.H + h) * (size_t)D * Dv + e0;
#pragma unroll 8
    for (int i = threadIdx.x; i < Dp * GC_EV; i += 256) {
        const int d = i / GC_EV, e = i % GC_EV;
        S[i] = d < D && e0 + e < Dv ? w[(size_t)d * Dv + e] : 0.f;
    }
    __syncthreads();
    const int ex = threadIdx.x & 15, ty = threadIdx.x >> 4;
    float acc[2][4] = {};
    auto rows = [&](const float* left, int ld, const float* right, int count) {
        for (int d = 0; d < count; d += 4) {
            const float4 l0 = *reinterpret_cast<const float4*>(left + ty * ld + d);
            const float4 l1 = *reinterpret_cast<const float4*>(left + (ty + 16) * ld + d);
#pragma unroll
            for (int y = 0; y < 4; ++y) {
                const float4 r = *reinterpret_cast<const float4*>(right + (d + y) * GC_EV + ex * 4);
                const float a0 = y == 0 ? l0.x : y == 1 ? l0.y : y == 2 ? l0.z : l0.w;
                const float a1 = y == 0 ? l1.x : y == 1 ? l1.y : y == 2 ? l1.z : l1.w;
                acc[0][0] = fmaf(a0, r.x, acc[0][0]); acc[0][1] = fmaf(a0, r.y, acc[0][1]);
                acc[0][2] = fmaf(a0, r.z, acc[0][2]); acc[0][3] = fmaf(a0, r.w, acc[0][3]);
                acc[1][0] = fmaf(a1, r.x, acc[1][0]); acc[1][1] = fmaf(a1, r.y, acc[1][1]);
                acc[1][2] = fmaf(a1, r.z, acc[1][2]); acc[1][3] = fmaf(a1, r.w, acc[1][3]);
            }
        }
    };
    rows(q, LD, S, Dp);
    rows(A, GC_LA, vs, GC_CHUNK);
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int t = ty + 16 * r;
        if (t >= n) break;
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (e0 + ex * 4 + u < Dv) a.out[(size_t)(t0 + t) * a.ldo + h * Dv + e0 + ex * 4 + u] = acc[r][u];
    }
}

static size_t gc_prep_smem(int D) {
    const size_t three = (size_t)3 * GC_CHUNK * gc_ld(D), sums = (size_t)GC_CHUNK * gc_ld(D) + 4 * GC_PAIRS * 64;
    return (three > sums ? three : sums) * sizeof(float);
}
static size_t gc_walk_smem(int D, int ev) {
    return ((size_t)2 * gc_floats(D) + (size_t)2 * gc_pad(D) * ev + 10 * GC_CHUNK * ev) * sizeof(float);
}

template <typename T, int EV, int DP>
static int launch_gated_walk_form(const GatedChunkArgs& c, int num_seqs, cudaStream_t st) {
    const int vz = (c.a.Dv + EV - 1) / EV;
    if (vz > 65535) return SLB_ERR_TOO_LARGE;
    static unsigned long long configured = 0;
    const int rc = slb_configure(&configured, gated_chunk_walk_kernel<T, EV, DP>, gc_walk_smem(GC_MAX_D, EV));
    if (rc != 0) return rc;
    return slb_launch_after(gated_chunk_walk_kernel<T, EV, DP>, dim3(num_seqs, c.a.H, vz), dim3(512),
                            gc_walk_smem(c.a.D, EV), st, c);
}
template <typename T, int EV>
static int launch_gated_walk(const GatedChunkArgs& c, int num_seqs, cudaStream_t st) {
    if (c.a.D == 128) return launch_gated_walk_form<T, EV, 128>(c, num_seqs, st);
    if (c.a.D == 64) return launch_gated_walk_form<T, EV, 64>(c, num_seqs, st);
    return launch_gated_walk_form<T, EV, 0>(c, num_seqs, st);
}

template <typename T>
static int launch_gated_parallel(const GatedChunkArgs& c, int num_seqs, cudaStream_t st) {
    const DecayAttnArgs& a = c.a;
    const int vz = (a.Dv + GC_EV - 1) / GC_EV, ez = (a.D * a.Dv + 255) / 256;
    if (vz > 65535 || ez > 65535) return SLB_ERR_TOO_LARGE;
    auto smem = [](int D, bool out) {
        return ((size_t)GC_CHUNK * (gc_ld(D) + GC_EV) + (out ? GC_CHUNK * GC_LA + gc_pad(D) * GC_EV : 0)) * sizeof(float);
    };
    static unsigned long long conf = 0;
    int rc = slb_configure(&conf, gated_chunk_out_kernel<T>, smem(GC_MAX_D, true));
    if (rc != 0) return rc;
    auto local = a.D <= 128 ? gated_chunk_local_kernel<T, 8> : gated_chunk_local_kernel<T, GC_MAX_D / 16>;
    rc = slb_launch(local, dim3(c.num_tiles, a.H, vz), dim3(256), smem(a.D, false), st, c);
    if (rc != 0) return rc;
    rc = slb_launch(gated_chunk_scan_kernel, dim3(num_seqs, a.H, ez), dim3(256), 0, st, c);
    if (rc != 0) return rc;
    return slb_launch(gated_chunk_out_kernel<T>, dim3(c.num_tiles, a.H, vz), dim3(256), smem(a.D, true), st, c);
}

template <typename T>
static int launch_gated_chunk(const GatedChunkArgs* c_in, int num_seqs, cudaStream_t st) {
    if (num_seqs <= 0 || c_in->num_tiles <= 0) return 0;
    GatedChunkArgs c = *c_in;
    DecayAttnArgs& a = c.a;
    if (a.state_stride <= 0) a.state_stride = (long long)a.H * a.D * a.Dv;
    if (a.H <= 0 || a.D <= 0 || a.Dv <= 0 || a.num_slots <= 0 || (a.rot_dims & 1) || a.rot_dims < 0 ||
        a.rot_dims > a.D || (a.rot_dims > 0 && a.freq == nullptr) || a.act < 0 || a.act > 1 ||
        a.gate_z == nullptr || a.ld_gate < a.H * a.D || !(a.gate_inv_tau > 0.f) || a.gate_kind < 0 ||
        a.gate_kind > 1 ||
        a.state_stride < (long long)a.H * a.D * a.Dv || c.work == nullptr || ((uintptr_t)c.work & 15) ||
        c.tile_seq == nullptr || c.tile_row0 == nullptr)
        return SLB_ERR_BAD_ARG;
    if (a.D > GC_MAX_D || a.H > 65535 || num_seqs > 65535) return SLB_ERR_TOO_LARGE;
    static unsigned long long conf1 = 0;
    int rc = slb_configure(&conf1, gated_chunk_prep_kernel<T>, gc_prep_smem(GC_MAX_D));
    if (rc != 0) return rc;
    rc = slb_launch(gated_chunk_prep_kernel<T>, dim3(c.num_tiles, a.H), dim3(256), gc_prep_smem(a.D), st, c);
    if (rc != 0) return rc;
    if (c.states != nullptr) return launch_gated_parallel<T>(c, num_seqs, st);
    // (the walk is serial in a request's chunks: while slices of 16 columns leave half of the SMs idle, slices of 8
    // share a chunk's work among twice as many: 512 tokens of 1 head of 128 x 128 34.6 us, 42.9 with 16; 1,024 +
    // 1,024 of 4 heads of 96 x 96 54 and 69; 256 of 4 heads of 64 x 128 18.3 and 20.6)
    const long long slices = (long long)num_seqs * a.H * ((a.Dv + 15) / 16);
    return 2 * slices < slb_num_sms() ? launch_gated_walk<T, 8>(c, num_seqs, st) : launch_gated_walk<T, 16>(c, num_seqs, st);
}

extern "C" {
int slb_decay_gated_chunk_max_dim() { return GC_MAX_D; }
int slb_decay_gated_chunk_tokens() { return GC_CHUNK; }
// 1: chunks of such a step are better worked on side by side (`states` is then wanted).  The walk costs 1.0 us a
// chunk of the longest request, the form without it two launches more, some 12 us, and the states' way through
// memory, 13 us for 2^20 elements.  Measured us walked / side by side, one request, by tokens: 4 heads of 64 x 128
// 2,048 75 / 52, 8,192 280 / 137; 2 of 64 x 64 1,024 41 / 26; 1 of 128 x 128 1,024 53 / 36, 8,192 316 / 104; 8 of
// 64 x 64 2,048 83 / 57; 8 of 128 x 256 2,048 145 / 224, 8,192 550 / 935 (the latter with a slower first launch).
// (The mean length stands for the longest: a step that is captured for later ones knows no more.)
int slb_decay_gated_chunk_side_by_side(int num_tiles, int num_seqs, int H, int D, int Dv) {
    const double chunks = (double)num_tiles / (num_seqs > 0 ? num_seqs : 1);
    return 0.95 * chunks > 14.0 + 13.0 / (1 << 20) * ((double)num_tiles * H * D * Dv);
}
int slb_decay_gated_chunk_work_floats(int D) { return gc_floats(D); }
int slb_decay_gated_chunk_f32(const GatedChunkArgs* c, int num_seqs, cudaStream_t st) {
    return launch_gated_chunk<float>(c, num_seqs, st);
}
int slb_decay_gated_chunk_bf16(const GatedChunkArgs* c, int num_seqs, cudaStream_t st) {
    return launch_gated_chunk<bf16>(c, num_seqs, st);
}
}

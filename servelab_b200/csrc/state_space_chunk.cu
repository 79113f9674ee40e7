// The selective state space (state_space.cu) for steps that bring portions of prompts, in its chunked form on
// the tensor cores (bf16 mma.sync, float32 accumulators).
//
// A request's portion is cut into chunks of 64 tokens from its first token on.  With S the state [N, P] that
// enters a chunk of n tokens, d_j the step sizes, L_i = -rate sum_{j <= i} d_j and i, j token indices in the chunk:
//
//     y_i   = e^(L_i) S^T C_i  +  sum_{j <= i} e^(L_i - L_j) d_j (C_i . B_j) x_j  +  skip x_i
//     S_out = e^(L_last) S     +  sum_j e^(L_last - L_j) d_j B_j x_j^T
//
// (all exponents are at most 0).  Two or three launches:
//
//   1. local sums   a block per (chunk, head, 64 value columns): sum_j e^(L_last - L_j) d_j B_j x_j^T, float32
//                   into a work buffer [chunks, H, N, P], and e^(L_last);
//   2. scan         a thread per some state elements of a (request, head): walks the request's chunks in
//                   order, leaves in the work buffer the state that ENTERS each chunk and the final state in
//                   the request's slot;
//   3. outputs      a block per chunk and some heads' value columns: the formula for y_i.
//
// State sizes of 64 and 128 have 1 and 2 in one launch while the requests are many or short: a walk over a
// request's chunks with the state in registers.
//
// x, B and C are bfloat16 as the convolution left them, so they are exact operands.  What is float32 -- the
// weighted x of launch 1, the weighted scores and the entering state of launch 3 -- is staged as two bfloat16
// numbers, hi = bf16(a) and lo = bf16(a - hi), two MMAs a product (an error of about 2^-17 of the product's terms).
// Step sizes, their sums, exponentials and the state are float32.
#include "mma_util.cuh"
#include "state_space.cuh"

using namespace slb_mma;

#define SC_CHUNK 64
#define SC_THREADS 256
#define SC_PAD 8                   // bf16 elements added to every shared row (ldmatrix without bank conflicts)
#define SC_MAX_N 256
#define SC_EV 64                   // value columns a block
#define SC_LDX (SC_EV + SC_PAD)
#define SC_SCAN_BATCH 8

struct StateSpaceChunkArgs {
    StateSpaceArgs a;
    const int* tile_seq; const int* tile_row0; int num_tiles;
    float* work;                   // [num_tiles][H][N][P]
    float* total;                  // [num_tiles][H]: e^(L_last)
};

// the chunk's first token and its number of tokens
__device__ __forceinline__ bool sc_tile(const StateSpaceChunkArgs& c, int tile, int& t0, int& n, int& s) {
    s = c.tile_seq[tile];
    const int q0 = c.a.cu_q[s], row0 = c.tile_row0[tile];
    n = min(SC_CHUNK, c.a.cu_q[s + 1] - q0 - row0);
    t0 = q0 + row0;
    return n > 0;
}

// step sizes and their running sums times -rate (one warp, two tokens a lane)
__device__ __forceinline__ void sc_steps_of(float d0, float d1, float rate, float* d, float* L) {
    const int lane = threadIdx.x & 31;
    float sum = d0 + d1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const float up = __shfl_up_sync(0xffffffffu, sum, o);
        if (lane >= o) sum += up;
    }
    const float before = sum - (d0 + d1);
    d[2 * lane] = d0;
    d[2 * lane + 1] = d1;
    L[2 * lane] = -rate * (before + d0);
    L[2 * lane + 1] = -rate * sum;
}
// (of the chunk's tokens; from n on: 0 and L_last)
__device__ __forceinline__ void sc_steps(const StateSpaceArgs& a, int h, int t0, int n, float* d, float* L) {
    const int lane = threadIdx.x & 31;
    const float bias = a.dt_bias[h], rate = a.rate[h];
    float d0 = 0.f, d1 = 0.f;
    if (2 * lane < n) d0 = ss_step(a.dt[(size_t)(t0 + 2 * lane) * a.ld_dt + h] + bias);
    if (2 * lane + 1 < n) d1 = ss_step(a.dt[(size_t)(t0 + 2 * lane + 1) * a.ld_dt + h] + bias);
    sc_steps_of(d0, d1, rate, d, L);
}

__device__ __forceinline__ void sc_zero(void* p, int bytes) {          // bytes a multiple of 16, p 16-byte aligned
    uint4* q = reinterpret_cast<uint4*>(p);
    for (int i = threadIdx.x; i < bytes / 16; i += SC_THREADS) q[i] = make_uint4(0, 0, 0, 0);
}

// `width` neighbouring elements of n rows, as they are
__device__ __forceinline__ void sc_stage(bf16* dst, int ldd, const bf16* src, int lds, int n, int width, bool wide) {
    if (wide) {
        const int wv = width >> 3;
        for (int idx = threadIdx.x; idx < n * wv; idx += SC_THREADS) {
            const int j = idx / wv, c = (idx - j * wv) << 3;
            *reinterpret_cast<uint4*>(dst + j * ldd + c) = *reinterpret_cast<const uint4*>(src + (size_t)j * lds + c);
        }
        return;
    }
    for (int idx = threadIdx.x; idx < n * width; idx += SC_THREADS) {
        const int j = idx / width, c = idx - j * width;
        dst[j * ldd + c] = src[(size_t)j * lds + c];
    }
}

// eight float32 numbers as hi and lo, `lo_off` elements apart
__device__ __forceinline__ void sc_put8(bf16* hi, int lo_off, int idx, const float (&x)[8]) {
    unsigned h[4], l[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        h[e] = pack_bf16(x[2 * e], x[2 * e + 1]);
        const __nv_bfloat162 hv = *reinterpret_cast<const __nv_bfloat162*>(&h[e]);
        l[e] = pack_bf16(x[2 * e] - __low2float(hv), x[2 * e + 1] - __high2float(hv));
    }
    *reinterpret_cast<uint4*>(hi + idx) = make_uint4(h[0], h[1], h[2], h[3]);
    *reinterpret_cast<uint4*>(hi + lo_off + idx) = make_uint4(l[0], l[1], l[2], l[3]);
}
__device__ __forceinline__ void sc_put(bf16* hi, int lo_off, int idx, float x) {
    const bf16 h = __float2bfloat16(x);
    hi[idx] = h;
    hi[lo_off + idx] = __float2bfloat16(x - __bfloat162float(h));
}

// rows of u whose pieces of 8 elements are whole 16-byte pieces
__device__ __forceinline__ bool sc_wide(const StateSpaceArgs& a) {
    return ((a.ld | a.x_off | a.b_off | a.c_off | a.P | a.N) & 7) == 0 && ((size_t)a.u & 15) == 0;
}

// State sizes of 64 and 128 with rows in whole 16-byte pieces have kernels of their own (NN).  What bounded them was no
// rate: two thirds of a block's time were the chain of loads that finds its chunk, the issue of its copies, and waits of
// the few warps an SM held; then the work buffer's three ways through memory.  A block of launch 3 takes several units,
// a unit being 64 value columns of a head, of one chunk and group: they share B and C, their scores C . B^T and that
// chain; the rows of the next unit arrive while one is worked on, and the entering state comes as the operand that the
// products take.  With the walk below, us before and now: 2,912 tokens of 4 requests, 32 heads of 128 x 64 103 -> 80; 64
// requests of 64 tokens 302 -> 98; 16 of 256 151 -> 77; one of 2,048 71 -> 55; one of 64 17.8 -> 13.6.
#define SC_MAX_UNITS 8

// A block's units: u-th of `count`, of group `grp`
struct StateUnits {
    int grp, first, count, slices, heads;                  // slices: of a head; heads: of a group
    __device__ __forceinline__ StateUnits(const StateSpaceArgs& a, int per_block) {
        slices = (a.P + SC_EV - 1) / SC_EV;
        heads = a.H / a.G;
        const int blocks = (heads * slices + per_block - 1) / per_block;
        grp = blockIdx.y / blocks;
        first = (blockIdx.y - grp * blocks) * per_block;
        count = min(per_block, heads * slices - first);
    }
    __device__ __forceinline__ int head(int u) const { return grp * heads + (first + u) / slices; }
    __device__ __forceinline__ int column(int u) const { return (first + u) % slices * SC_EV; }
};

template <int WV>
__device__ __forceinline__ void sc_stage_async(bf16* dst, int ldd, const bf16* src, int lds, int n, int width) {
#pragma unroll
    for (int idx = threadIdx.x; idx < SC_CHUNK * WV; idx += SC_THREADS) {
        const int j = idx / WV, col = (idx % WV) * 8;
        const bool ok = j < n && col < width;
        cp_async16(dst + j * ldd + col, src + (ok ? (size_t)j * lds + col : 0), ok);
    }
}

// ------------------------------------------------------------------ 1. local sums of a chunk
// sum_j B_j xw_j^T of the staged rows: the weighted x as hi and lo, into dst [N][P]
__device__ __forceinline__ void sc_local_products(const bf16* bs, int ldn, const bf16* xs, float* dst, int N, int P, int e0,
                                                  int width, int n) {
    constexpr int x_elems = SC_CHUNK * SC_LDX;
    const int Np = (N + 15) & ~15;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int ksteps = (n + 15) >> 4;
    const bool pairs = !(P & 1);
    for (int unit = warp; unit < Np / 8; unit += SC_THREADS / 32) {       // 16 state rows x 32 value columns
        const int mt = unit >> 1, half = unit & 1;
        if (half * 32 >= width) continue;
        float acc[4][4];
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
        for (int kk = 0; kk < ksteps; ++kk) {
            // A[m = n][k = token] from rows stored [token][n]
            unsigned af[4];
            ldmatrix_x4_trans(af, bs + (kk * 16 + (lane & 7) + ((lane >> 4) & 1) * 8) * ldn + mt * 16 + ((lane >> 3) & 1) * 8);
#pragma unroll
            for (int np = 0; np < 2; ++np) {
                // B[k = token][n = e] from rows stored [token][e]
                const int b_at = (kk * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * SC_LDX + half * 32 + np * 16 +
                                 ((lane >> 4) & 1) * 8;
                unsigned bh[4], bl[4];
                ldmatrix_x4_trans(bh, xs + b_at);
                ldmatrix_x4_trans(bl, xs + x_elems + b_at);
                mma_bf16(acc[2 * np], af, bl[0], bl[1]);
                mma_bf16(acc[2 * np + 1], af, bl[2], bl[3]);
                mma_bf16(acc[2 * np], af, bh[0], bh[1]);
                mma_bf16(acc[2 * np + 1], af, bh[2], bh[3]);
            }
        }
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
            const int e = e0 + half * 32 + nt * 8 + 2 * t;
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const int row = mt * 16 + g + r * 8;
                if (row >= N) continue;
                float* o = dst + (size_t)row * P + e;
                if (pairs && e + 1 < P) {
                    *reinterpret_cast<float2*>(o) = make_float2(acc[nt][2 * r], acc[nt][2 * r + 1]);
                } else {
                    if (e < P) o[0] = acc[nt][2 * r];
                    if (e + 1 < P) o[1] = acc[nt][2 * r + 1];
                }
            }
        }
    }
}

__global__ void __launch_bounds__(SC_THREADS) state_chunk_local_kernel(const StateSpaceChunkArgs c) {
    extern __shared__ __align__(16) unsigned char sc_smem[];
    __shared__ float d[SC_CHUNK], L[SC_CHUNK];
    pdl_wait();
    pdl_launch_dependents();
    const StateSpaceArgs& a = c.a;
    const int tile = blockIdx.x, h = blockIdx.y, e0 = blockIdx.z * SC_EV;
    int t0, n, s;
    if (!sc_tile(c, tile, t0, n, s)) return;
    const int N = a.N, P = a.P, Np = (N + 15) & ~15, ldn = Np + SC_PAD;
    const int width = min(SC_EV, P - e0), grp = h / (a.H / a.G);
    const int x_elems = SC_CHUNK * SC_LDX;
    bf16* bs = reinterpret_cast<bf16*>(sc_smem);           // [64][ldn]
    bf16* xs = bs + SC_CHUNK * ldn;                        // [hi, lo][64][SC_LDX]
    const bf16* u = reinterpret_cast<const bf16*>(a.u) + (size_t)t0 * a.ld;
    const bf16* x = u + a.x_off + h * P + e0;
    if (n < SC_CHUNK || N < Np || width < SC_EV) {  // (a full tile is written whole)
        sc_zero(bs, (SC_CHUNK * ldn + 2 * x_elems) * (int)sizeof(bf16));
    }
    if (threadIdx.x < 32) sc_steps(a, h, t0, n, d, L);
    __syncthreads();
    const bool wide = sc_wide(a);
    const float last = L[SC_CHUNK - 1];
    if (threadIdx.x == 0 && e0 == 0) c.total[(size_t)tile * a.H + h] = decay_exp(last);
    sc_stage(bs, ldn, u + a.b_off + grp * N, a.ld, n, N, wide);
    if (wide) {
        const int wv = width >> 3;
        for (int idx = threadIdx.x; idx < n * wv; idx += SC_THREADS) {
            const int j = idx / wv, col = (idx - j * wv) << 3;
            const uint4 raw = *reinterpret_cast<const uint4*>(x + (size_t)j * a.ld + col);
            const unsigned w[4] = {raw.x, raw.y, raw.z, raw.w};
            const float f = d[j] * expf(last - L[j]);
            float v[8];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float2 p = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w[e]));
                v[2 * e] = p.x * f;
                v[2 * e + 1] = p.y * f;
            }
            sc_put8(xs, x_elems, j * SC_LDX + col, v);
        }
    } else {
        for (int idx = threadIdx.x; idx < n * width; idx += SC_THREADS) {
            const int j = idx / width, col = idx - j * width;
            sc_put(xs, x_elems, j * SC_LDX + col, to_float(x[(size_t)j * a.ld + col]) * d[j] * expf(last - L[j]));
        }
    }
    __syncthreads();

    sc_local_products(bs, ldn, xs, c.work + ((size_t)tile * a.H + h) * (size_t)N * P, N, P, e0, width, n);
}

// ------------------------------------------------------------------ 2. the states that enter the chunks
// A request's chunks are neighbours in the tile list, in order.  What bounds it is the work buffer, read and
// written: three blocks an SM with the loads of eight chunks in flight (of sixteen with one block, and every
// thread with the exponentials and the search of its own: 31 us for 48 chunks of 32 heads of 128 x 64).
template <int V>
__global__ void __launch_bounds__(256, 3) state_chunk_scan_kernel(const StateSpaceChunkArgs c) {
    pdl_wait();
    pdl_launch_dependents();
    const StateSpaceArgs& a = c.a;
    const int s = blockIdx.x, h = blockIdx.y;
    const int qlen = a.cu_q[s + 1] - a.cu_q[s];
    if (qlen <= 0) return;
    const int slot = a.state_slots[s];
    if (slot < 0 || slot >= a.num_slots) return;
    const int elems = a.N * a.P;
    const int idx = (blockIdx.z * blockDim.x + threadIdx.x) * V;
    __shared__ int first_s;
    if (threadIdx.x == 0) first_s = c.num_tiles;
    __syncthreads();
    for (int i = threadIdx.x; i < c.num_tiles; i += 256)
        if (c.tile_seq[i] == s) { atomicMin(&first_s, i); break; }
    __syncthreads();
    if (idx >= elems) return;
    const int first = first_s;
    const int count = (qlen + SC_CHUNK - 1) / SC_CHUNK;
    if (first + count > c.num_tiles) return;
    float* sp = a.state + (size_t)slot * (size_t)a.state_stride + (size_t)h * elems + idx;
    float* wp = c.work + ((size_t)first * a.H + h) * (size_t)elems + idx;
    const float* lp = c.total + (size_t)first * a.H + h;
    const size_t step = (size_t)a.H * elems;
    float S[V];
    auto load = [](const float* p, float (&v)[V]) {
        if constexpr (V == 4) {
            const float4 x = *reinterpret_cast<const float4*>(p);
            v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
        } else {
            v[0] = p[0];
        }
    };
    auto store = [](float* p, const float (&v)[V]) {
        if constexpr (V == 4) *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
        else p[0] = v[0];
    };
    load(sp, S);
    // (the loads of a batch do not wait for one another: one memory latency a batch, not a chunk)
    for (int k0 = 0; k0 < count; k0 += SC_SCAN_BATCH) {
        float add[SC_SCAN_BATCH][V], g[SC_SCAN_BATCH];
#pragma unroll
        for (int b = 0; b < SC_SCAN_BATCH; ++b) {
            const bool in = k0 + b < count;
            if (in) load(wp + b * step, add[b]);
            g[b] = in ? lp[(size_t)(k0 + b) * a.H] : 0.f;
        }
#pragma unroll
        for (int b = 0; b < SC_SCAN_BATCH; ++b) {
            if (k0 + b < count) {
                store(wp + b * step, S);
#pragma unroll
                for (int v = 0; v < V; ++v) S[v] = fmaf(g[b], S[v], add[b][v]);
            }
        }
        wp += SC_SCAN_BATCH * step;
    }
    store(sp, S);
}

// acc[state row / 8] += the chunk's weighted x (16 columns from 16 et on) by B (NT tiles of 8 state rows from n0 on)
template <int NT>
__device__ __forceinline__ void sc_walk_products(const bf16* xs, const bf16* bs, int ldb, const float* weight, int et, int n0,
                                                 int lane, float (&acc)[NT][4]) {
    const int t = lane & 3;
#pragma unroll
    for (int kk = 0; kk < SC_CHUNK / 16; ++kk) {
        // A[m = e][k = token] from rows stored [token][e], weighted and split
        unsigned raw[4], ah[4], al[4];
        ldmatrix_x4_trans(raw, xs + (kk * 16 + (lane & 7) + ((lane >> 4) & 1) * 8) * SC_LDX + et * 16 + ((lane >> 3) & 1) * 8);
        const float2 w0 = *reinterpret_cast<const float2*>(weight + kk * 16 + 2 * t);
        const float2 w1 = *reinterpret_cast<const float2*>(weight + kk * 16 + 8 + 2 * t);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const float2 v = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw[r]));
            const float x0 = v.x * (r < 2 ? w0.x : w1.x), x1 = v.y * (r < 2 ? w0.y : w1.y);
            ah[r] = pack_bf16(x0, x1);
            const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&ah[r]));
            al[r] = pack_bf16(x0 - f.x, x1 - f.y);
        }
#pragma unroll
        for (int j = 0; j < NT / 2; ++j) {
            // B[k = token][n = state row] from rows stored [token][n]
            unsigned bf[4];
            ldmatrix_x4_trans(bf, bs + (kk * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * ldb + n0 + j * 16 + ((lane >> 4) & 1) * 8);
            mma_bf16(acc[2 * j], al, bf[0], bf[1]);
            mma_bf16(acc[2 * j + 1], al, bf[2], bf[3]);
            mma_bf16(acc[2 * j], ah, bf[0], bf[1]);
            mma_bf16(acc[2 * j + 1], ah, bf[2], bf[3]);
        }
    }
}

// The state as launch 3 takes it: of 16 columns x 16 state rows a lane has 8 numbers, in the order b0, b1 of columns 0..7
// (state rows 2t, 2t + 1 and 8 more), b0, b1 of columns 8..15; their hi are 16 bytes, their lo lie 32 lanes on.
__device__ __forceinline__ void sc_put_tile(uint4* w, const float (&v)[8]) {
    unsigned hi[4], lo[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        hi[r] = pack_bf16(v[2 * r], v[2 * r + 1]);
        const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&hi[r]));
        lo[r] = pack_bf16(v[2 * r] - f.x, v[2 * r + 1] - f.y);
    }
    w[0] = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    w[32] = make_uint4(lo[0], lo[1], lo[2], lo[3]);
}

// ------------------------------------------------------------------ 1 and 2 in one: a walk over a request's chunks
// Rows in whole 16-byte pieces: a block per (request, head, 64 value columns, NB state rows) keeps its part of the state
// in registers and takes the request's chunks in order.  The products are formed with the value columns as the rows of the
// accumulators: what a lane then holds of 16 columns x 16 state rows is what launch 3 needs as its B operand, and
// goes to the work buffer as that, hi and lo, 16 bytes a lane.  Three chunks of x and B are on their way; the
// steps and weights, a chain of 1,300 cycles a chunk, are formed for sixteen chunks at a time by all warps.  Per chunk:
// work [head][P / 16][N / 16][hi, lo][32 lanes] of 16 bytes.
#define SC_WALK_STAGES 3
#define SC_WALK_BATCH 16
template <int NB>
__global__ void __launch_bounds__(SC_THREADS, 2) state_chunk_walk_kernel(const StateSpaceChunkArgs c) {
    extern __shared__ __align__(16) unsigned char sc_smem[];
    __shared__ float d[8][SC_CHUNK], L[8][SC_CHUNK], weight[SC_WALK_BATCH][SC_CHUNK];
    __shared__ float decay[SC_WALK_BATCH];
    __shared__ int first_s;
    pdl_wait();
    pdl_launch_dependents();
    constexpr int LDB = NB + SC_PAD, XE = SC_CHUNK * SC_LDX, STAGE = XE + SC_CHUNK * LDB;
    constexpr int NT = NB / 16;                            // tiles of 8 state rows a warp
    const StateSpaceArgs& a = c.a;
    const int s = blockIdx.x, h = blockIdx.y, parts = a.N / NB, part = blockIdx.z % parts, e0 = blockIdx.z / parts * SC_EV;
    const int q0 = a.cu_q[s], qlen = a.cu_q[s + 1] - q0;
    const int slot = a.state_slots[s];
    if (qlen <= 0 || slot < 0 || slot >= a.num_slots) return;
    if (threadIdx.x == 0) first_s = c.num_tiles;
    __syncthreads();
    for (int i = threadIdx.x; i < c.num_tiles; i += SC_THREADS)
        if (c.tile_seq[i] == s) { atomicMin(&first_s, i); break; }
    const int P = a.P, width = min(SC_EV, P - e0), count = (qlen + SC_CHUNK - 1) / SC_CHUNK;
    bf16* stages = reinterpret_cast<bf16*>(sc_smem);       // [3]: [64][SC_LDX] of x, [64][LDB] of B
    const bf16* u = reinterpret_cast<const bf16*>(a.u) + (size_t)q0 * a.ld;
    const bf16* x = u + a.x_off + h * P + e0;
    const bf16* B = u + a.b_off + h / (a.H / a.G) * a.N + part * NB;
    // a thread's pieces of a chunk: x of tokens tj and tj + 32, and of B every BROWS tokens from bj on
    constexpr int BROWS = SC_THREADS / (NB / 8);
    const int tj = threadIdx.x >> 3, tcol = (threadIdx.x & 7) * 8, bj = threadIdx.x / (NB / 8), bcol = threadIdx.x % (NB / 8) * 8;
    const bf16* x_at = x + (size_t)tj * a.ld + tcol;
    const bf16* b_at = B + (size_t)bj * a.ld + bcol;
    int asked = 0, ask_stage = 0;                          // tokens of the chunks asked for, the next one's place
    auto ask = [&]() {
        if (asked < qlen) {
            bf16* st = stages + ask_stage * STAGE;
            const int n = qlen - asked;
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const bool ok = tj + q * 32 < n && tcol < width;
                cp_async16(st + (tj + q * 32) * SC_LDX + tcol, ok ? x_at + (size_t)q * 32 * a.ld : x, ok);
            }
#pragma unroll
            for (int q = 0; q < SC_CHUNK / BROWS; ++q) {
                const bool ok = bj + q * BROWS < n;
                cp_async16(st + XE + (bj + q * BROWS) * LDB + bcol, ok ? b_at + (size_t)q * BROWS * a.ld : B, ok);
            }
            x_at += (size_t)SC_CHUNK * a.ld;
            b_at += (size_t)SC_CHUNK * a.ld;
        }
        asked += SC_CHUNK;
        ask_stage = ask_stage == SC_WALK_STAGES - 1 ? 0 : ask_stage + 1;
        cp_async_commit();
    };
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const float bias = a.dt_bias[h], rate = a.rate[h];
    auto weights = [&](int k0) {                           // of the chunks from k0 on, two a warp
        for (int b = warp; b < SC_WALK_BATCH && k0 + b < count; b += 8) {
            const int n = qlen - (k0 + b) * SC_CHUNK;
            const float* dt = a.dt + (size_t)(q0 + (k0 + b) * SC_CHUNK + 2 * lane) * a.ld_dt + h;
            sc_steps_of(2 * lane < n ? ss_step(dt[0] + bias) : 0.f, 2 * lane + 1 < n ? ss_step(dt[a.ld_dt] + bias) : 0.f, rate,
                        d[warp], L[warp]);
            __syncwarp();
            const float last = L[warp][SC_CHUNK - 1];
#pragma unroll
            for (int j = lane; j < SC_CHUNK; j += 32) weight[b][j] = d[warp][j] * expf(last - L[warp][j]);
            if (lane == 0) decay[b] = decay_exp(last);
            __syncwarp();
        }
    };
    ask();
    ask();
    weights(0);

    const int et = warp & 3, n0 = (warp >> 2) * (NB / 2);  // this warp's 16 columns, its first state row of the part
    const bool live = et * 16 < width;
    float S[NT][4];
    float* sp = a.state + (size_t)slot * (size_t)a.state_stride + (size_t)h * a.N * P;
    auto at = [&](int nt, int r) {                         // (columns of 16 that are not there: 0, not stored)
        const int e = e0 + et * 16 + g + 8 * (r >> 1), n = part * NB + n0 + nt * 8 + 2 * t + (r & 1);
        return live && e < P ? sp + (size_t)n * P + e : nullptr;
    };
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const float* p = at(nt, r);
            S[nt][r] = p ? *p : 0.f;
        }
    __syncthreads();
    const int first = first_s;
    if (first + count > c.num_tiles) {
        cp_async_wait<0>();
        return;
    }
    const int etiles = (P + 15) >> 4, ntiles = a.N >> 4;
    uint4* work = reinterpret_cast<uint4*>(c.work) +
                  ((((size_t)first * a.H + h) * etiles + (e0 >> 4) + et) * ntiles + ((part * NB + n0) >> 4)) * 64 + lane;
    const size_t step = (size_t)a.H * etiles * ntiles * 64;
    for (int k = 0, stage = 0; k < count; ++k, stage = stage == SC_WALK_STAGES - 1 ? 0 : stage + 1) {
        cp_async_wait<1>();
        __syncthreads();                                   // the chunk is there; every warp is done with the one before
        ask();
        const int b = k % SC_WALK_BATCH;
        if (b == 0 && k > 0) {
            weights(k);
            __syncthreads();
        }
        if (!live) continue;
        uint4* w = work + (size_t)k * step;
#pragma unroll
        for (int j = 0; j < NT / 2; ++j) {
            const float v[8] = {S[2 * j][0], S[2 * j][1], S[2 * j + 1][0], S[2 * j + 1][1],
                                S[2 * j][2], S[2 * j][3], S[2 * j + 1][2], S[2 * j + 1][3]};
            sc_put_tile(w + j * 64, v);
        }
        const bf16* xs = stages + stage * STAGE;
        const bf16* bs = xs + XE;
        float acc[NT][4];
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
        sc_walk_products<NT>(xs, bs, LDB, weight[b], et, n0, lane, acc);
        const float f = decay[b];
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int r = 0; r < 4; ++r) S[nt][r] = fmaf(f, S[nt][r], acc[nt][r]);
    }
    if (!live) return;
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            float* p = at(nt, r);
            if (p) *p = S[nt][r];
        }
}

// The same with the chunks side by side, for few and long requests: the sums of every chunk, float32 in the places of the
// hi and lo, and a scan that a thread walks with the 8 numbers of a lane.
template <int NN>
__global__ void __launch_bounds__(SC_THREADS, 2) state_chunk_sums_kernel(const StateSpaceChunkArgs c) {
    extern __shared__ __align__(16) unsigned char sc_smem[];
    __shared__ float d[SC_CHUNK], L[SC_CHUNK], weight[SC_CHUNK];
    pdl_wait();
    pdl_launch_dependents();
    constexpr int LDB = NN + SC_PAD, NT = NN / 16;
    const StateSpaceArgs& a = c.a;
    const int tile = blockIdx.x, h = blockIdx.y, e0 = blockIdx.z * SC_EV, P = a.P, width = min(SC_EV, P - e0);
    int t0, n, s;
    if (!sc_tile(c, tile, t0, n, s)) return;
    bf16* xs = reinterpret_cast<bf16*>(sc_smem);           // [64][SC_LDX]
    bf16* bs = xs + SC_CHUNK * SC_LDX;                     // [64][LDB]
    const bf16* u = reinterpret_cast<const bf16*>(a.u) + (size_t)t0 * a.ld;
    sc_stage_async<SC_EV / 8>(xs, SC_LDX, u + a.x_off + h * P + e0, a.ld, n, width);
    sc_stage_async<NN / 8>(bs, LDB, u + a.b_off + h / (a.H / a.G) * NN, a.ld, n, NN);
    cp_async_commit();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp == 0) {
        sc_steps(a, h, t0, n, d, L);
        __syncwarp();
        const float last = L[SC_CHUNK - 1];
#pragma unroll
        for (int j = lane; j < SC_CHUNK; j += 32) weight[j] = d[j] * expf(last - L[j]);
        if (lane == 0 && e0 == 0) c.total[(size_t)tile * a.H + h] = decay_exp(last);
    }
    cp_async_wait<0>();
    __syncthreads();
    const int et = warp & 3, n0 = (warp >> 2) * (NN / 2);
    if (et * 16 >= width) return;
    float acc[NT][4];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
    sc_walk_products<NT>(xs, bs, LDB, weight, et, n0, lane, acc);
    float4* w = reinterpret_cast<float4*>(c.work) +
                ((((size_t)tile * a.H + h) * ((P + 15) >> 4) + (e0 >> 4) + et) * (NN / 16) + (n0 >> 4)) * 64 + lane;
#pragma unroll
    for (int j = 0; j < NT / 2; ++j) {
        w[j * 64] = make_float4(acc[2 * j][0], acc[2 * j][1], acc[2 * j + 1][0], acc[2 * j + 1][1]);
        w[j * 64 + 32] = make_float4(acc[2 * j][2], acc[2 * j][3], acc[2 * j + 1][2], acc[2 * j + 1][3]);
    }
}

// What bounds it is what an SM takes in and gives back, 2 KB a chunk and tile: blocks of two tiles, so that few heads have
// many SMs (blocks of eight: 9.5 us for 32 chunks of 8 heads of 64 x 32, 6.7 now).
#define SC_TILE_BATCH 8
#define SC_TILE_THREADS 64
__global__ void __launch_bounds__(SC_TILE_THREADS, 8) state_chunk_scan_tiles_kernel(const StateSpaceChunkArgs c) {
    pdl_wait();
    pdl_launch_dependents();
    const StateSpaceArgs& a = c.a;
    const int s = blockIdx.x, h = blockIdx.y, P = a.P, etiles = (P + 15) >> 4, ntiles = a.N >> 4;
    const int qlen = a.cu_q[s + 1] - a.cu_q[s], slot = a.state_slots[s];
    if (qlen <= 0 || slot < 0 || slot >= a.num_slots) return;
    __shared__ int first_s;
    if (threadIdx.x == 0) first_s = c.num_tiles;
    __syncthreads();
    for (int i = threadIdx.x; i < c.num_tiles; i += SC_TILE_THREADS)
        if (c.tile_seq[i] == s) { atomicMin(&first_s, i); break; }
    __syncthreads();
    const int first = first_s, count = (qlen + SC_CHUNK - 1) / SC_CHUNK;
    const int tile = (blockIdx.z * SC_TILE_THREADS + threadIdx.x) >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    if (tile >= etiles * ntiles || first + count > c.num_tiles) return;
    float* sp = a.state + (size_t)slot * (size_t)a.state_stride + (size_t)h * a.N * P;
    auto at = [&](int i) {                                 // (columns that are not there: 0, not stored)
        const int e = tile / ntiles * 16 + g + 8 * (i >> 2), n = tile % ntiles * 16 + 8 * (i >> 1 & 1) + 2 * t + (i & 1);
        return e < P ? sp + (size_t)n * P + e : nullptr;
    };
    float S[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) S[i] = at(i) ? *at(i) : 0.f;
    const size_t step = (size_t)a.H * etiles * ntiles * 64;
    uint4* w = reinterpret_cast<uint4*>(c.work) + (((size_t)first * a.H + h) * etiles * ntiles + tile) * 64 + lane;
    const float* lp = c.total + (size_t)first * a.H + h;
    for (int k0 = 0; k0 < count; k0 += SC_TILE_BATCH) {
        float4 add[SC_TILE_BATCH][2];
        float f[SC_TILE_BATCH];
#pragma unroll
        for (int b = 0; b < SC_TILE_BATCH; ++b) {
            const bool in = k0 + b < count;
            if (in) {
                add[b][0] = *reinterpret_cast<const float4*>(w + b * step);
                add[b][1] = *reinterpret_cast<const float4*>(w + b * step + 32);
            }
            f[b] = in ? lp[(size_t)(k0 + b) * a.H] : 0.f;
        }
#pragma unroll
        for (int b = 0; b < SC_TILE_BATCH; ++b) {
            if (k0 + b < count) {
                sc_put_tile(w + b * step, S);
                const float v[8] = {add[b][0].x, add[b][0].y, add[b][0].z, add[b][0].w,
                                    add[b][1].x, add[b][1].y, add[b][1].z, add[b][1].w};
#pragma unroll
                for (int i = 0; i < 8; ++i) S[i] = fmaf(f[b], S[i], v[i]);
            }
        }
        w += SC_TILE_BATCH * step;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
        if (at(i)) *at(i) = S[i];
}

// ------------------------------------------------------------------ 3. the chunk's outputs
// a warp's 16 tokens x 32 columns: the products and skip x
__device__ __forceinline__ void sc_store(const StateSpaceArgs& a, const bf16* xs, const float (&acc)[4][4], int t0, int n, int h,
                                         int e0, int wc, int i0, int t) {
    const int P = a.P;
    const float skip = a.skip[h];
    const bool pairs = !((P | a.ldo) & 1);
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
        const int ec = (wc * 4 + nt) * 8 + 2 * t, e = e0 + ec;
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int i = i0 + half * 8;
            if (i >= n) continue;
            const bf16* xr = xs + i * SC_LDX + ec;
            const float y0 = fmaf(skip, to_float(xr[0]), acc[nt][2 * half]);
            const float y1 = fmaf(skip, to_float(xr[1]), acc[nt][2 * half + 1]);
            float* o = a.out + (size_t)(t0 + i) * a.ldo + (size_t)h * P + e;
            if (pairs && e + 1 < P) {
                *reinterpret_cast<float2*>(o) = make_float2(y0, y1);
            } else {
                if (e < P) o[0] = y0;
                if (e + 1 < P) o[1] = y1;
            }
        }
    }
}

// Eight warps: 16 tokens and 32 of the value columns each (the scores of 16 tokens are formed by the two warps
// that share them).  The weighted scores stay in registers: the accumulator of C . B^T of 16 tokens x 16 tokens
// has the layout of the A operand of the product with x.  The entering state takes the place of B once the
// scores are formed.
__global__ void __launch_bounds__(SC_THREADS, 2) state_chunk_out_kernel(const StateSpaceChunkArgs c) {
    extern __shared__ __align__(16) unsigned char sc_smem[];
    __shared__ float d[SC_CHUNK], L[SC_CHUNK];
    pdl_wait();
    pdl_launch_dependents();
    const StateSpaceArgs& a = c.a;
    const int tile = blockIdx.x, h = blockIdx.y, e0 = blockIdx.z * SC_EV;
    int t0, n, s;
    if (!sc_tile(c, tile, t0, n, s)) return;
    const int slot = a.state_slots[s];
    if (slot < 0 || slot >= a.num_slots) return;
    const int N = a.N, P = a.P, Np = (N + 15) & ~15, ldn = Np + SC_PAD;
    const int width = min(SC_EV, P - e0), grp = h / (a.H / a.G);
    const int n_elems = SC_CHUNK * ldn, s_elems = Np * SC_LDX;
    bf16* cs = reinterpret_cast<bf16*>(sc_smem);           // [64][ldn]
    bf16* xs = cs + n_elems;                               // [64][SC_LDX]
    bf16* bs = xs + SC_CHUNK * SC_LDX;                     // [64][ldn], later [hi, lo][Np][SC_LDX]
    const bf16* u = reinterpret_cast<const bf16*>(a.u) + (size_t)t0 * a.ld;
    const float* entering = c.work + ((size_t)tile * a.H + h) * (size_t)N * P + e0;
    if (n < SC_CHUNK || N < Np || width < SC_EV)
        sc_zero(cs, (n_elems + SC_CHUNK * SC_LDX + n_elems) * (int)sizeof(bf16));
    if (threadIdx.x < 32) sc_steps(a, h, t0, n, d, L);
    __syncthreads();
    const bool wide = sc_wide(a);
    sc_stage(cs, ldn, u + a.c_off + grp * N, a.ld, n, N, wide);
    sc_stage(bs, ldn, u + a.b_off + grp * N, a.ld, n, N, wide);
    sc_stage(xs, SC_LDX, u + a.x_off + h * P + e0, a.ld, n, width, wide);
    __syncthreads();

    const int warp = (threadIdx.x >> 5) & 3, wc = threadIdx.x >> 7;     // token group, half of the columns
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const bool live = warp * 16 < n && wc * 32 < width;
    const int a_row = (warp * 16 + (lane & 15)) * ldn + ((lane >> 4) & 1) * 8;   // A[m = token][k = n], + kk * 16
    const int i0 = warp * 16 + g;                           // this lane's two tokens: i0, i0 + 8

    float p[8][4];
#pragma unroll
    for (int nt = 0; nt < 8; ++nt) p[nt][0] = p[nt][1] = p[nt][2] = p[nt][3] = 0.f;
    if (live) {
        for (int kk = 0; kk < Np / 16; ++kk) {
            unsigned af[4];
            ldmatrix_x4(af, cs + a_row + kk * 16);
#pragma unroll
            for (int np = 0; np < 4; ++np) {
                if (np <= warp) {
                    // B[k = n][n = token] from rows stored [token][n]
                    unsigned bf[4];
                    ldmatrix_x4(bf, bs + (np * 16 + (lane & 7) + ((lane >> 4) & 1) * 8) * ldn + kk * 16 + ((lane >> 3) & 1) * 8);
                    mma_bf16(p[2 * np], af, bf[0], bf[1]);
                    mma_bf16(p[2 * np + 1], af, bf[2], bf[3]);
                }
            }
        }
        const float L0 = L[i0], L1 = L[i0 + 8];
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
            if (nt <= 2 * warp + 1) {
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const int i = i0 + 8 * (r >> 1), j = nt * 8 + 2 * t + (r & 1);
                    p[nt][r] = (j <= i && i < n) ? p[nt][r] * (d[j] * expf((r >> 1 ? L1 : L0) - L[j])) : 0.f;
                }
            }
        }
    }
    __syncthreads();                                        // every warp is done with B

    // the entering state's tile [n][e] over it (padding rows and columns zero)
    const float* src = entering;
    if (N < Np || width < SC_EV) {
        sc_zero(bs, 2 * s_elems * (int)sizeof(bf16));
        __syncthreads();
    }
    if ((P & 7) == 0) {
        const int wv = width >> 3;
#pragma unroll 4
        for (int idx = threadIdx.x; idx < N * wv; idx += SC_THREADS) {
            const int row = idx / wv, col = (idx - row * wv) << 3;
            const float4 u0 = *reinterpret_cast<const float4*>(src + (size_t)row * P + col);
            const float4 u1 = *reinterpret_cast<const float4*>(src + (size_t)row * P + col + 4);
            const float v[8] = {u0.x, u0.y, u0.z, u0.w, u1.x, u1.y, u1.z, u1.w};
            sc_put8(bs, s_elems, row * SC_LDX + col, v);
        }
    } else {
        for (int idx = threadIdx.x; idx < N * width; idx += SC_THREADS) {
            const int row = idx / width, col = idx - row * width;
            sc_put(bs, s_elems, row * SC_LDX + col, src[(size_t)row * P + col]);
        }
    }
    __syncthreads();
    if (!live) return;                                      // (no barrier follows)

    float acc[4][4];
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
    for (int kk = 0; kk < Np / 16; ++kk) {
        unsigned af[4];
        ldmatrix_x4(af, cs + a_row + kk * 16);
#pragma unroll
        for (int np = 0; np < 2; ++np) {
            // B[k = n][n = e] from rows stored [n][e]
            const int b_at = (kk * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * SC_LDX + (wc * 2 + np) * 16 + ((lane >> 4) & 1) * 8;
            unsigned bh[4], bl[4];
            ldmatrix_x4_trans(bh, bs + b_at);
            ldmatrix_x4_trans(bl, bs + s_elems + b_at);
            mma_bf16(acc[2 * np], af, bl[0], bl[1]);
            mma_bf16(acc[2 * np], af, bh[0], bh[1]);
            mma_bf16(acc[2 * np + 1], af, bl[2], bl[3]);
            mma_bf16(acc[2 * np + 1], af, bh[2], bh[3]);
        }
    }
    {
        const float f0 = expf(L[i0]), f1 = expf(L[i0 + 8]);
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
            acc[nt][0] *= f0; acc[nt][1] *= f0;
            acc[nt][2] *= f1; acc[nt][3] *= f1;
        }
    }
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
        if (kk <= warp) {
            unsigned ah[4], al[4];
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const float x0 = p[2 * kk + (r >> 1)][2 * (r & 1)], x1 = p[2 * kk + (r >> 1)][2 * (r & 1) + 1];
                ah[r] = pack_bf16(x0, x1);
                const __nv_bfloat162 hv = *reinterpret_cast<const __nv_bfloat162*>(&ah[r]);
                al[r] = pack_bf16(x0 - __low2float(hv), x1 - __high2float(hv));
            }
#pragma unroll
            for (int np = 0; np < 2; ++np) {
                // B[k = token][n = e] from rows stored [token][e]
                unsigned bf[4];
                ldmatrix_x4_trans(bf, xs + (kk * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * SC_LDX + (wc * 2 + np) * 16 +
                                          ((lane >> 4) & 1) * 8);
                mma_bf16(acc[2 * np], al, bf[0], bf[1]);
                mma_bf16(acc[2 * np], ah, bf[0], bf[1]);
                mma_bf16(acc[2 * np + 1], al, bf[2], bf[3]);
                mma_bf16(acc[2 * np + 1], ah, bf[2], bf[3]);
            }
        }
    }
    sc_store(a, xs, acc, t0, n, h, e0, wc, i0, t);
}

// The same for several units of a chunk and group.  The scores of 16 tokens stay in registers as they are and are
// weighted for each unit; the two warps of a scheduler take the first and the last of the token groups, whose numbers of
// scores differ by four.
template <int NN>
__global__ void __launch_bounds__(SC_THREADS, 2) state_chunk_out_units_kernel(const StateSpaceChunkArgs c, int per_block) {
    extern __shared__ __align__(16) unsigned char sc_smem[];
    __shared__ float d[SC_MAX_UNITS][SC_CHUNK], L[SC_MAX_UNITS][SC_CHUNK];
    pdl_wait();
    pdl_launch_dependents();
    const StateSpaceArgs& a = c.a;
    const int tile = blockIdx.x, P = a.P, etiles = (P + 15) >> 4;
    int t0, n, s;
    if (!sc_tile(c, tile, t0, n, s)) return;
    constexpr int LDN = NN + SC_PAD, ST = 2 * NN * SC_EV, BUF = ST + SC_CHUNK * SC_LDX;
    const StateUnits units(a, per_block);
    bf16* cs = reinterpret_cast<bf16*>(sc_smem);           // [64][LDN]
    bf16* bufs = cs + SC_CHUNK * LDN;                      // two units: the state as the walk left it, [64][SC_LDX] of x
    bf16* bs = bufs + BUF;                                 // [64][LDN] in the second buffer until the scores are formed
    const bf16* u = reinterpret_cast<const bf16*>(a.u) + (size_t)t0 * a.ld;
    auto ask = [&](int unit) {
        const int h = units.head(unit), e0 = units.column(unit), width = min(SC_EV, P - e0);
        bf16* buf = bufs + (unit & 1) * BUF;
        const bf16* entering = reinterpret_cast<const bf16*>(c.work) + (((size_t)tile * a.H + h) * etiles + (e0 >> 4)) * (NN * 32);
        const int pieces = min(4, etiles - (e0 >> 4)) * NN * 4;
#pragma unroll
        for (int q = 0; q < NN * 16 / SC_THREADS; ++q) {
            const int idx = threadIdx.x + q * SC_THREADS;
            if (idx < pieces) cp_async16(buf + idx * 8, entering + idx * 8, true);
        }
        sc_stage_async<SC_EV / 8>(buf + ST, SC_LDX, u + a.x_off + h * P + e0, a.ld, n, width);
        cp_async_commit();
    };
    sc_stage_async<NN / 8>(cs, LDN, u + a.c_off + units.grp * NN, a.ld, n, NN);
    sc_stage_async<NN / 8>(bs, LDN, u + a.b_off + units.grp * NN, a.ld, n, NN);
    cp_async_commit();
    const int slot = a.state_slots[s];
    const bool present = slot >= 0 && slot < a.num_slots;
    if (present) ask(0);
    if ((threadIdx.x >> 5) < units.count)
        sc_steps(a, units.head(threadIdx.x >> 5), t0, n, d[threadIdx.x >> 5], L[threadIdx.x >> 5]);
    if (!present) {
        cp_async_wait<0>();
        return;
    }
    cp_async_wait<1>();
    __syncthreads();

    const int wc = threadIdx.x >> 7, warp = wc ? 3 - ((threadIdx.x >> 5) & 3) : (threadIdx.x >> 5) & 3;
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int a_row = (warp * 16 + (lane & 15)) * LDN + ((lane >> 4) & 1) * 8;
    const int i0 = warp * 16 + g;

    float p[8][4];
#pragma unroll
    for (int nt = 0; nt < 8; ++nt) p[nt][0] = p[nt][1] = p[nt][2] = p[nt][3] = 0.f;
    if (warp * 16 < n) {
#pragma unroll 2
        for (int kk = 0; kk < NN / 16; ++kk) {
            unsigned af[4];
            ldmatrix_x4(af, cs + a_row + kk * 16);
#pragma unroll
            for (int np = 0; np < 4; ++np) {
                if (np <= warp) {
                    unsigned bf[4];
                    ldmatrix_x4(bf, bs + (np * 16 + (lane & 7) + ((lane >> 4) & 1) * 8) * LDN + kk * 16 + ((lane >> 3) & 1) * 8);
                    mma_bf16(p[2 * np], af, bf[0], bf[1]);
                    mma_bf16(p[2 * np + 1], af, bf[2], bf[3]);
                }
            }
        }
    }
    for (int unit = 0; unit < units.count; ++unit) {
        cp_async_wait<0>();
        __syncthreads();                                   // the unit is there; every warp is done with the one before (and B)
        if (unit + 1 < units.count) ask(unit + 1);
        const int h = units.head(unit), e0 = units.column(unit), width = min(SC_EV, P - e0);
        if (warp * 16 >= n || wc * 32 >= width) continue;
        const bf16* st = bufs + (unit & 1) * BUF;
        const bf16* xs = st + ST;
        const float* du = d[unit];
        const float* Lu = L[unit];
        float acc[4][4];
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
#pragma unroll 2
        for (int kk = 0; kk < NN / 16; ++kk) {
            unsigned af[4];
            ldmatrix_x4(af, cs + a_row + kk * 16);
#pragma unroll
            for (int np = 0; np < 2; ++np) {
                // B[k = n][n = e], in the lanes' order
                const bf16* tile_at = st + ((wc * 2 + np) * (NN / 16) + kk) * 512 + lane * 8;
                const uint4 bh = *reinterpret_cast<const uint4*>(tile_at), bl = *reinterpret_cast<const uint4*>(tile_at + 256);
                mma_bf16(acc[2 * np], af, bl.x, bl.y);
                mma_bf16(acc[2 * np + 1], af, bl.z, bl.w);
                mma_bf16(acc[2 * np], af, bh.x, bh.y);
                mma_bf16(acc[2 * np + 1], af, bh.z, bh.w);
            }
        }
        const float L0 = Lu[i0], L1 = Lu[i0 + 8];
        const float f0 = expf(L0), f1 = expf(L1);
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
            acc[nt][0] *= f0; acc[nt][1] *= f0;
            acc[nt][2] *= f1; acc[nt][3] *= f1;
        }
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
            if (kk <= warp) {
                unsigned ah[4], al[4];
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const int i = i0 + 8 * (r & 1), j = (2 * kk + (r >> 1)) * 8 + 2 * t;
                    const float2 dj = *reinterpret_cast<const float2*>(du + j), Lj = *reinterpret_cast<const float2*>(Lu + j);
                    const float Li = (r & 1) ? L1 : L0;
                    const float* raw = p[2 * kk + (r >> 1)] + 2 * (r & 1);
                    const float x0 = (j <= i && i < n) ? raw[0] * (dj.x * expf(Li - Lj.x)) : 0.f;
                    const float x1 = (j + 1 <= i && i < n) ? raw[1] * (dj.y * expf(Li - Lj.y)) : 0.f;
                    ah[r] = pack_bf16(x0, x1);
                    const __nv_bfloat162 hv = *reinterpret_cast<const __nv_bfloat162*>(&ah[r]);
                    al[r] = pack_bf16(x0 - __low2float(hv), x1 - __high2float(hv));
                }
#pragma unroll
                for (int np = 0; np < 2; ++np) {
                    unsigned bf[4];
                    ldmatrix_x4_trans(bf, xs + (kk * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * SC_LDX + (wc * 2 + np) * 16 +
                                              ((lane >> 4) & 1) * 8);
                    mma_bf16(acc[2 * np], al, bf[0], bf[1]);
                    mma_bf16(acc[2 * np + 1], al, bf[2], bf[3]);
                    mma_bf16(acc[2 * np], ah, bf[0], bf[1]);
                    mma_bf16(acc[2 * np + 1], ah, bf[2], bf[3]);
                }
            }
        }
        sc_store(a, xs, acc, t0, n, h, e0, wc, i0, t);
    }
}

static size_t sc_local_smem(int N) {
    const int Np = (N + 15) & ~15;
    return ((size_t)SC_CHUNK * (Np + SC_PAD) + 2 * SC_CHUNK * SC_LDX) * sizeof(bf16);
}
static size_t sc_out_smem(int N) {
    const int Np = (N + 15) & ~15;
    const size_t rows = (size_t)SC_CHUNK * (Np + SC_PAD), st = (size_t)2 * Np * SC_LDX;
    return (rows + SC_CHUNK * SC_LDX + (rows > st ? rows : st)) * sizeof(bf16);
}
static size_t sc_out_units_smem(int N) {
    return ((size_t)SC_CHUNK * (N + SC_PAD) + (size_t)2 * (2 * N * SC_EV + SC_CHUNK * SC_LDX)) * sizeof(bf16);
}

// Units a block, for `tiles` chunks and `resident` blocks a multiprocessor: the fewest rounds of blocks, a round
// counted as its units and about one more for what the block does before its first.
static int sc_units(const StateSpaceArgs& a, int tiles, int resident) {
    const int units = a.H / a.G * ((a.P + SC_EV - 1) / SC_EV), sms = slb_num_sms();
    long long best_cost = 0;
    int best = 1;
    for (int k = 1; k <= SC_MAX_UNITS && k <= units; ++k) {
        const long long blocks = (long long)tiles * a.G * ((units + k - 1) / k);
        const long long rounds = (blocks + (long long)sms * resident - 1) / ((long long)sms * resident), cost = rounds * (k + 1);
        if (best_cost == 0 || cost < best_cost) best_cost = cost, best = k;
    }
    return best;
}

template <int NB>
static int launch_state_walk(const StateSpaceChunkArgs& c, int num_seqs, int slices, cudaStream_t st) {
    static unsigned long long done = 0;
    const size_t smem = (size_t)SC_WALK_STAGES * SC_CHUNK * (SC_LDX + NB + SC_PAD) * sizeof(bf16);
    const int rc = slb_configure(&done, state_chunk_walk_kernel<NB>, smem);
    if (rc != 0) return rc;
    return slb_launch(state_chunk_walk_kernel<NB>, dim3(num_seqs, c.a.H, slices * (c.a.N / NB)), dim3(SC_THREADS), smem, st, c);
}

// Whether a step takes the kernels for rows in whole pieces (NN), and whether these have the chunks side by side.  The walk
// is a chain of about 0.9 us a chunk of the longest request; the chunks side by side take a launch more and the states' way
// through memory twice more (us walked / side by side, state size x values, heads: 64 x 32, 8, 320 / 384 / 512 / 2,048 tokens
// 12.4 / 12.6, 13.1 / 12.4, 14.5 / 12.6, 33.6 / 18.0; 64 x 64, 32, 512 / 1,024 / 2,048 21.6 / 17.7, 36.0 / 23.2, 64.7 / 37.8, 64
// heads 25.4 / 22.7, 43.6 / 36.2, 80.3 / 63.9; 128 x 64, 32, 256 / 512 / 768 / 1,024 / 2,048 18.3 / 18.8, 23.6 / 22.0, 33.6 / 29.5,
// 38.8 / 33.0, 69.1 / 53.5, 64 heads 19.4 / 20.3, 29.1 / 30.2, 39.6 / 39.9, 49.3 / 49.4, 90.9 / 92.9; 4 x 512 of 32 heads 41.9 /
// 50.8, 16 x 400 121 / 179).
static bool sc_in_pieces(const StateSpaceArgs& a) {
    return ((a.ld | a.x_off | a.b_off | a.c_off | a.P) & 7) == 0 && ((uintptr_t)a.u & 15) == 0 &&
           (long long)a.H * ((a.P + SC_EV - 1) / SC_EV) <= 65535 && (a.N == 64 || a.N == 128);
}
static bool sc_side_by_side(const StateSpaceChunkArgs& c, int num_seqs, int longest) {
    const StateSpaceArgs& a = c.a;
    const int chunks = longest > 0 ? (longest + SC_CHUNK - 1) / SC_CHUNK : (c.num_tiles + num_seqs - 1) / num_seqs;
    const int slices = (a.P + SC_EV - 1) / SC_EV;
    return 0.9 * chunks > 4.7 + 0.009 / 8192 * ((double)c.num_tiles * a.H * slices * SC_EV * a.N);
}

template <int NN>
static int launch_state_chunks(const StateSpaceChunkArgs& c, int num_seqs, int longest, cudaStream_t st) {
    static unsigned long long done = 0;
    const StateSpaceArgs& a = c.a;
    int rc = slb_configure(&done, state_chunk_out_units_kernel<NN>, sc_out_units_smem(NN));
    if (rc != 0) return rc;
    const int slices = (a.P + SC_EV - 1) / SC_EV, units = a.H / a.G * slices, per = sc_units(a, c.num_tiles, 2);
    const long long whole = (long long)num_seqs * a.H * slices, room = 2 * slb_num_sms();
    if (sc_side_by_side(c, num_seqs, longest)) {
        static unsigned long long done_sums = 0;
        const size_t smem = (size_t)SC_CHUNK * (SC_LDX + NN + SC_PAD) * sizeof(bf16);
        rc = slb_configure(&done_sums, state_chunk_sums_kernel<NN>, smem);
        if (rc == 0) rc = slb_launch(state_chunk_sums_kernel<NN>, dim3(c.num_tiles, a.H, slices), dim3(SC_THREADS), smem, st, c);
        const int tiles = (a.P + 15) / 16 * (NN / 16);
        if (rc == 0) rc = slb_launch(state_chunk_scan_tiles_kernel, dim3(num_seqs, a.H, (tiles + 1) / 2), dim3(SC_TILE_THREADS), 0, st, c);
    } else if (whole * (NN / 32) <= room) {                // (the finest cut whose blocks are all resident)
        rc = launch_state_walk<32>(c, num_seqs, slices, st);
    } else if (NN == 64 || whole * (NN / 64) <= room) {
        rc = launch_state_walk<64>(c, num_seqs, slices, st);
    } else {
        rc = launch_state_walk<128>(c, num_seqs, slices, st);
    }
    if (rc != 0) return rc;
    return slb_launch(state_chunk_out_units_kernel<NN>, dim3(c.num_tiles, a.G * ((units + per - 1) / per)), dim3(SC_THREADS),
                      sc_out_units_smem(NN), st, c, per);
}

extern "C" {
int slb_state_space_chunk_tokens() { return SC_CHUNK; }
// kernels that slb_state_space_chunk_bf16 launches for the same arguments
int slb_state_space_chunk_launches(const StateSpaceChunkArgs* c, int num_seqs, int longest) {
    if (num_seqs <= 0 || c->num_tiles <= 0) return 0;
    return sc_in_pieces(c->a) && !sc_side_by_side(*c, num_seqs, longest) ? 2 : 3;
}
// u bfloat16; the tile list cuts every request's tokens of the step into chunks of slb_state_space_chunk_tokens()
// (request, first row), a request's in order.
// work: num_tiles x H x N x (P rounded up to 16) numbers; longest: tokens of the longest request (0: not known, the mean
// stands for it).
int slb_state_space_chunk_bf16(const StateSpaceChunkArgs* c, int num_seqs, int longest, cudaStream_t st) {
    const StateSpaceArgs& a = c->a;
    if (num_seqs <= 0 || c->num_tiles <= 0) return 0;
    if (a.H <= 0 || a.P <= 0 || a.N <= 0 || a.G <= 0 || a.H % a.G != 0 || a.num_slots <= 0 ||
        a.state_stride < (long long)a.H * a.N * a.P || a.ldo < a.H * a.P || a.ld_dt < a.H || c->work == nullptr ||
        c->total == nullptr || c->tile_seq == nullptr || c->tile_row0 == nullptr ||
        (((uintptr_t)c->work | (uintptr_t)a.out) & 15))
        return SLB_ERR_BAD_ARG;
    if (a.N > SC_MAX_N || a.H > 65535 || a.P > 65535) return SLB_ERR_TOO_LARGE;
    const int elems = a.N * a.P;
    const bool quads = elems % 4 == 0 && a.state_stride % 4 == 0 && ((uintptr_t)a.state & 15) == 0;
    if (sc_in_pieces(a))
        return a.N == 128 ? launch_state_chunks<128>(*c, num_seqs, longest, st) : launch_state_chunks<64>(*c, num_seqs, longest, st);
    static unsigned long long done_local = 0, done_out = 0;
    int rc = slb_configure(&done_local, state_chunk_local_kernel, sc_local_smem(SC_MAX_N));
    if (rc == 0) rc = slb_configure(&done_out, state_chunk_out_kernel, sc_out_smem(SC_MAX_N));
    if (rc != 0) return rc;
    const dim3 grid(c->num_tiles, a.H, (a.P + SC_EV - 1) / SC_EV);
    rc = slb_launch(state_chunk_local_kernel, grid, dim3(SC_THREADS), sc_local_smem(a.N), st, *c);
    if (rc != 0) return rc;
    if (quads)
        rc = slb_launch(state_chunk_scan_kernel<4>, dim3(num_seqs, a.H, (elems / 4 + 255) / 256), dim3(256), 0, st, *c);
    else
        rc = slb_launch(state_chunk_scan_kernel<1>, dim3(num_seqs, a.H, (elems + 255) / 256), dim3(256), 0, st, *c);
    if (rc != 0) return rc;
    return slb_launch(state_chunk_out_kernel, grid, dim3(SC_THREADS), sc_out_smem(a.N), st, *c);
}
}

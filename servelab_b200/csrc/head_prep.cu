// What happens to the projected queries, keys and values of a step between the product and the
// attention, for mixers that norm heads and rotate neighbouring pairs:
//
//   optional biases on the projected queries, keys and values (rows of H * Dq, G * Dk, G * Dv);
//   optional RMS norm of ALL query heads of a token together, and of all key heads (`row_norm`), with a
//   weight for every element of the row;
//   per query head and per key head (a "vector" of D elements of the product's row):
//     * RMS norm over its first `norm_dims` elements with a weight shared by the heads
//       (x / sqrt(mean(x^2) + eps) * w; 0: no norm);
//     * rotation of `rot_dims` elements starting at `rot_off`: element 2i is paired with element
//       2i + 1 (or, with `rot_half`, element i with element i + rot_dims / 2), the pair (u, v) at
//       position p becomes (u c - v s, v c + u s) with
//       c = mag cos(p f_i), s = mag sin(p f_i) (a table of frequencies, one factor on both);
//     * after the rotation, division of the first `unit_dims` elements by their root mean square
//       (no weight; 0: none);
//     * queries go to the q buffer -- head h at h * q_head_stride, without its first `q_skip`
//       elements (a latent attention replaces them by their product with a matrix and keeps the
//       rotated rest) --, keys into the request's page (block-table look-up here);
//   per value head (optional):
//     * v <- (1 - lambda) v + lambda v_first with the values another layer computed for the same
//       token (optional), or a copy of v kept for the layers that will ask for it;
//     * into the request's page.
//
// The same kernel serves a grouped-query attention (queries and keys normed over the whole head
// and rotated from element 0) and a latent attention (one "key" of latent + rotated part: norm
// over the latent, rotation of the rest; queries rotated from `rot_off` on, not normed).
// One block a token (and group of vectors), one warp a vector at a time; the token's sines and
// cosines are formed once a block; float32 arithmetic, angles in float32.
#include <type_traits>

#include "gated_act.cuh"

#define HP_WARPS 4
#define HP_MAX_D 1152

SLB_DEFINE_STATUS_WORD(head_prep_status_word, slb_head_prep_status)

struct HeadPrepArgs {
    const void* proj; int ld;
    int q_off, H, Dq, q_norm_dims, q_rot_off; const float* q_norm_w;
    int k_off, G, Dk, k_norm_dims, k_rot_off; const float* k_norm_w;
    int v_off, Dv;
    const float* lambda; const void* v_first; int ld_vf; void* v_keep; int ld_vk;
    const float* freq; int rot_dims; float rot_mag; float eps;
    const int* positions; const int* seq_of_token; const int* block_table;
    int max_pages, page_size, num_pages;
    void* q_out; int ldq; void* k_cache; void* v_cache;
    int q_head_stride, q_skip;
    int rot_half, q_unit_dims, k_unit_dims;
    const float* q_bias; const float* k_bias; const float* v_bias;     // or null
    int row_norm;                  // the norm weights q_norm_w, k_norm_w then have H * Dq and G * Dk elements
};

// sum of squares of n elements (+ bias) of a row over the block; the order depends on n alone
template <typename T>
__device__ __forceinline__ float row_square_sum(const T* row, const float* bias, int n, float* scratch) {
    float ss = 0.f;
    for (int i = threadIdx.x; i < n; i += HP_WARPS * 32) {
        const float v = to_float(row[i]) + (bias != nullptr ? bias[i] : 0.f);
        ss += v * v;
    }
    return block_sum(ss, scratch);
}

template <typename T>
__global__ void __launch_bounds__(HP_WARPS * 32) head_prep_kernel(const HeadPrepArgs a) {
    extern __shared__ float hp_smem[];
    pdl_wait();
    pdl_launch_dependents();
    const int t = blockIdx.x;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int maxd = max(max(a.Dq, a.Dk), a.Dv);
    float* buf = hp_smem + (size_t)warp * maxd;
    float* cs_tab = hp_smem + (size_t)HP_WARPS * maxd;     // cos and sin of the token's angles, once a block
    float* sn_tab = cs_tab + a.rot_dims / 2;
    const T* row = reinterpret_cast<const T*>(a.proj) + (size_t)t * a.ld;
    const int pos = a.positions[t];
    for (int i = threadIdx.x; i < a.rot_dims / 2; i += blockDim.x) {
        float sn, cs;
        sincosf((float)pos * a.freq[i], &sn, &cs);
        cs_tab[i] = cs * a.rot_mag;
        sn_tab[i] = sn * a.rot_mag;
    }
    __shared__ float scratch[33];
    float q_rstd = 1.f, k_rstd = 1.f;
    if (a.row_norm) {
        q_rstd = 1.0f / sqrtf(row_square_sum(row + a.q_off, a.q_bias, a.H * a.Dq, scratch) / (float)(a.H * a.Dq) + a.eps);
        k_rstd = 1.0f / sqrtf(row_square_sum(row + a.k_off, a.k_bias, a.G * a.Dk, scratch) / (float)(a.G * a.Dk) + a.eps);
    }
    __syncthreads();
    // where this token's key and value go
    long long slot = -1;
    if (a.k_cache != nullptr || a.v_cache != nullptr) {
        const int page = a.block_table[(size_t)a.seq_of_token[t] * a.max_pages + pos / a.page_size];
        if (page >= a.num_pages) {
            if (lane == 0) atomicCAS(&head_prep_status_word, 0, 1);
        } else if (page >= 0) {
            slot = (long long)page * a.G * a.page_size + pos % a.page_size;
        }
    }
    const int nv = a.v_off >= 0 ? a.G : 0;
    const int units = a.H + a.G + nv;
    // (grid y: groups of HP_WARPS vectors, so that a step of few tokens still fills the device)
    for (int u = blockIdx.y * HP_WARPS + warp; u < units; u += gridDim.y * HP_WARPS) {
        const T* src;
        T* dst = nullptr;
        int D, norm_dims = 0, rot_off = 0, unit_dims = 0;
        const float* nw = nullptr;
        const float* bias = nullptr;                   // of this vector
        float rstd = 1.f;
        bool rotate = a.rot_dims > 0;
        int vhead = -1, skip = 0;
        if (u < a.H) {
            D = a.Dq; norm_dims = a.q_norm_dims; nw = a.q_norm_w; rot_off = a.q_rot_off; unit_dims = a.q_unit_dims;
            src = row + a.q_off + (size_t)u * D;
            dst = reinterpret_cast<T*>(a.q_out) + (size_t)t * a.ldq + (size_t)u * a.q_head_stride;
            skip = a.q_skip;
            if (a.q_bias != nullptr) bias = a.q_bias + (size_t)u * D;
            if (a.row_norm) { rstd = q_rstd; nw += (size_t)u * D; }
        } else if (u < a.H + a.G) {
            const int g = u - a.H;
            D = a.Dk; norm_dims = a.k_norm_dims; nw = a.k_norm_w; rot_off = a.k_rot_off; unit_dims = a.k_unit_dims;
            src = row + a.k_off + (size_t)g * D;
            if (a.k_bias != nullptr) bias = a.k_bias + (size_t)g * D;
            if (a.row_norm) { rstd = k_rstd; nw += (size_t)g * D; }
            if (a.k_cache != nullptr && slot >= 0)
                dst = reinterpret_cast<T*>(a.k_cache) + (size_t)(slot + (long long)g * a.page_size) * D;
        } else {
            vhead = u - a.H - a.G;
            D = a.Dv; rotate = false;
            src = row + a.v_off + (size_t)vhead * D;
            if (a.v_bias != nullptr) bias = a.v_bias + (size_t)vhead * D;
            if (a.v_cache != nullptr && slot >= 0)
                dst = reinterpret_cast<T*>(a.v_cache) + (size_t)(slot + (long long)vhead * a.page_size) * D;
        }
        __syncwarp();
        for (int i = lane; i < D; i += 32) buf[i] = to_float(src[i]) + (bias != nullptr ? bias[i] : 0.f);
        __syncwarp();
        if (vhead >= 0) {
            if (a.v_keep != nullptr) {
                T* keep = reinterpret_cast<T*>(a.v_keep) + (size_t)t * a.ld_vk + (size_t)vhead * D;
                for (int i = lane; i < D; i += 32) keep[i] = from_float<T>(buf[i]);
            }
            if (a.v_first != nullptr) {
                const float lam = a.lambda[0];
                const T* vf = reinterpret_cast<const T*>(a.v_first) + (size_t)t * a.ld_vf + (size_t)vhead * D;
                for (int i = lane; i < D; i += 32) buf[i] = (1.0f - lam) * buf[i] + lam * to_float(vf[i]);
            }
        } else {
            if (a.row_norm) {
                for (int i = lane; i < D; i += 32) buf[i] = buf[i] * rstd * nw[i];
            } else if (norm_dims > 0) {
                float ss = 0.f;
                for (int i = lane; i < norm_dims; i += 32) ss += buf[i] * buf[i];
                ss = warp_sum(ss);
                const float r = 1.0f / sqrtf(ss / (float)norm_dims + a.eps);
                for (int i = lane; i < norm_dims; i += 32) buf[i] = buf[i] * r * (nw != nullptr ? nw[i] : 1.f);
            }
            if (rotate) {
                __syncwarp();                          // (the norm wrote elements other lanes rotate)
                const int half = a.rot_dims / 2;
                for (int i = lane; i < half; i += 32) {
                    const float sn = sn_tab[i], cs = cs_tab[i];
                    const int ix = a.rot_half ? rot_off + i : rot_off + 2 * i;
                    const int iy = a.rot_half ? rot_off + i + half : rot_off + 2 * i + 1;
                    const float x = buf[ix], y = buf[iy];
                    buf[ix] = x * cs - y * sn;
                    buf[iy] = y * cs + x * sn;
                }
            }
            if (unit_dims > 0) {
                __syncwarp();
                float ss = 0.f;
                for (int i = lane; i < unit_dims; i += 32) ss += buf[i] * buf[i];
                ss = warp_sum(ss);
                const float r = 1.0f / sqrtf(ss / (float)unit_dims + a.eps);
                for (int i = lane; i < unit_dims; i += 32) buf[i] *= r;
            }
        }
        __syncwarp();
        if (dst != nullptr)
            for (int i = skip + lane; i < D; i += 32) dst[i - skip] = from_float<T>(buf[i]);
    }
}

// ---- bfloat16 rows in whole 16-byte pieces ------------------------------------------------------
// The same steps with the vectors in registers: a lane holds 8 neighbouring elements (one 16-byte
// load), as many lanes as a vector needs hold it (its sums are shuffles, a pair of halves is a
// shuffle, a pair of neighbours is in one lane), so a warp works on several short vectors at once
// and a thread has all its loads in flight before the sines are formed.  What bounds both kernels is
// the number of instructions (this one issues in half of the cycles), not memory.  Measured, general
// kernel against this one, us: 2,048 tokens of 16 + 4 + 4 heads of 128, half rotated, unit norms 23.7 ->
// 14.6; 2,912 tokens of 16 + 4 heads of 128 and 4 of 64, norms over the rows, biases 28.0 -> 18.5; 2,082
// tokens of a latent attention (16 queries of 192, of which 64 are read, a key of 320) 21.0 -> 12.7;
// 64 single tokens of 16 + 4 + 4 heads of 128 3.8 -> 3.4.
#define HPV_ITEMS 4          // vectors (of a lane) that are loaded together

struct HeadPrepKind {
    int off, stride;         // first element in the projected row; elements from one vector to the next
    int pieces, shift;       // 16-byte pieces of a vector; 1 << shift lanes hold it
    int units, items;        // vectors; warps' worth of vectors
    int norm, rot, unit;     // pieces that are normed, first piece that is rotated, pieces of the unit norm
    int skip;                // pieces that are not written
};
struct HeadPrepPlan { HeadPrepKind kind[3]; int items; };

__device__ __forceinline__ void unpack8(const uint4 r, float* v) {
    const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        v[2 * i] = __uint_as_float(w[i] << 16);
        v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
}
__device__ __forceinline__ uint4 pack8(const float* v) {
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
        w[i] = *reinterpret_cast<const uint32_t*>(&h);
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
}
// (weights and biases: read-only for every kernel of a step, so these loads may pass stores)
__device__ __forceinline__ void load8_weights(const float* p, float* v) {
    const float4 a = __ldg(reinterpret_cast<const float4*>(p)), b = __ldg(reinterpret_cast<const float4*>(p) + 1);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
__device__ __forceinline__ float lanes_sum(float v, int shift) {
    for (int o = (1 << shift) >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float square8(const float* v) {
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) s += v[i] * v[i];
    return s;
}

// PIECES: 16-byte pieces of a vector a lane may hold (2: vectors of more than 256 elements).  ROW: all
// heads of a token are normed together (one round and one block then hold the whole token).  DENSE: a third more
// warps an SM, with some registers spilled (the launch decides).
template <int PIECES, bool ROW, bool DENSE>
__global__ void __launch_bounds__(256, (PIECES == 1 ? 3 : 2) + (DENSE ? 1 : 0)) head_prep_vec_kernel(
    const __grid_constant__ HeadPrepArgs a, const __grid_constant__ HeadPrepPlan p) {
    extern __shared__ __align__(16) float hp_smem[];
    __shared__ float2 row_part[8];
    float* cs_tab = hp_smem;                              // of the token's angles, once a block
    float* sn_tab = cs_tab + a.rot_dims / 2;
    const int t = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    const int q_items = p.kind[0].items, qk_items = q_items + p.kind[1].items;
    pdl_wait();
    pdl_launch_dependents();
    const bf16* row = reinterpret_cast<const bf16*>(a.proj) + (size_t)t * a.ld;
    const int step = warps * gridDim.y;
    const int pos = a.positions[t];
    int page = -1;                                        // where this token's key and value go
    for (int first = blockIdx.y * warps + warp, round = 0; round * HPV_ITEMS * step < p.items;
         ++round, first += HPV_ITEMS * step) {
        uint4 raw[HPV_ITEMS][PIECES];
        int kind[HPV_ITEMS], unit[HPV_ITEMS];
#pragma unroll
        for (int j = 0; j < HPV_ITEMS; ++j) {
            const int item = first + j * step;
            const int k = (item >= q_items) + (item >= qk_items);
            const HeadPrepKind& kd = p.kind[k];
            const int at = item - (k == 0 ? 0 : k == 1 ? q_items : qk_items);
            kind[j] = k;
            unit[j] = item < p.items ? (at << (5 - kd.shift)) + (lane >> kd.shift) : 0x7fffffff;
            const int l = lane & ((1 << kd.shift) - 1);
#pragma unroll
            for (int c = 0; c < PIECES; ++c) {
                const int piece = l + c * 32;
                raw[j][c] = make_uint4(0, 0, 0, 0);
                if (unit[j] < kd.units && piece < kd.pieces)
                    raw[j][c] = *reinterpret_cast<const uint4*>(row + kd.off + unit[j] * kd.stride + piece * 8);
            }
        }
        if (round == 0) {                                 // (its lookup waits for two loads: behind the row's)
            if (a.k_cache != nullptr || a.v_cache != nullptr)
                page = a.block_table[(size_t)a.seq_of_token[t] * a.max_pages + pos / a.page_size];
            for (int i = threadIdx.x; i < a.rot_dims / 2; i += blockDim.x) {
                float sn, cs;
                sincosf((float)pos * a.freq[i], &sn, &cs);
                cs_tab[i] = cs * a.rot_mag;
                sn_tab[i] = sn * a.rot_mag;
            }
        }
        float q_rstd = 1.f, k_rstd = 1.f;
        if (ROW) {
            float ss[2] = {0.f, 0.f};
#pragma unroll
            for (int j = 0; j < HPV_ITEMS; ++j) {
                if (kind[j] == 2) continue;
                const HeadPrepKind& kd = p.kind[kind[j]];
                const int l = lane & ((1 << kd.shift) - 1);
                const float* bias = kind[j] == 0 ? a.q_bias : a.k_bias;
                float sum = 0.f;
#pragma unroll
                for (int c = 0; c < PIECES; ++c) {
                    const int piece = l + c * 32;
                    if (unit[j] >= kd.units || piece >= kd.pieces) continue;
                    float v[8], b[8];
                    unpack8(raw[j][c], v);
                    if (bias != nullptr) {
                        load8_weights(bias + unit[j] * kd.stride + piece * 8, b);
#pragma unroll
                        for (int e = 0; e < 8; ++e) v[e] += b[e];
                    }
                    sum += square8(v);
                }
                if (kind[j] == 0) ss[0] += sum; else ss[1] += sum;
            }
            ss[0] = warp_sum(ss[0]);
            ss[1] = warp_sum(ss[1]);
            if (lane == 0) row_part[warp] = make_float2(ss[0], ss[1]);
        }
        if (ROW || (a.rot_dims > 0 && round == 0)) __syncthreads();
        if (ROW) {
            float qs = 0.f, ks = 0.f;
            for (int i = 0; i < warps; ++i) {
                qs += row_part[i].x;
                ks += row_part[i].y;
            }
            q_rstd = 1.0f / sqrtf(qs / (float)(a.H * a.Dq) + a.eps);
            k_rstd = 1.0f / sqrtf(ks / (float)(a.G * a.Dk) + a.eps);
        }
        long long slot = -1;
        if (page >= a.num_pages) {
            if (lane == 0 && (a.k_cache != nullptr || a.v_cache != nullptr)) atomicCAS(&head_prep_status_word, 0, 1);
        } else if (page >= 0) {
            slot = (long long)page * a.G * a.page_size + pos % a.page_size;
        }
#pragma unroll
        for (int j = 0; j < HPV_ITEMS; ++j) {
            if (first + j * step >= p.items) break;
            const int k = kind[j], u = unit[j];
            const HeadPrepKind& kd = p.kind[k];
            const int l = lane & ((1 << kd.shift) - 1);
            const float* bias = k == 0 ? a.q_bias : k == 1 ? a.k_bias : a.v_bias;
            bf16* dst = nullptr;
            if (u < kd.units) {
                if (k == 0)
                    dst = reinterpret_cast<bf16*>(a.q_out) + (size_t)t * a.ldq + u * a.q_head_stride;
                else if (slot >= 0 && k == 1 && a.k_cache != nullptr)
                    dst = reinterpret_cast<bf16*>(a.k_cache) + (size_t)(slot + (long long)u * a.page_size) * a.Dk;
                else if (slot >= 0 && k == 2 && a.v_cache != nullptr)
                    dst = reinterpret_cast<bf16*>(a.v_cache) + (size_t)(slot + (long long)u * a.page_size) * a.Dv;
            }
            float v[PIECES][8];
#pragma unroll
            for (int c = 0; c < PIECES; ++c) {
                const int piece = l + c * 32;
                unpack8(raw[j][c], v[c]);
                if (bias != nullptr && u < kd.units && piece < kd.pieces) {
                    float b[8];
                    load8_weights(bias + u * kd.stride + piece * 8, b);
#pragma unroll
                    for (int e = 0; e < 8; ++e) v[c][e] += b[e];
                }
            }
            if (k == 2) {
                if (a.v_keep != nullptr || a.v_first != nullptr) {
#pragma unroll
                    for (int c = 0; c < PIECES; ++c) {
                        const int piece = l + c * 32;
                        if (u >= kd.units || piece >= kd.pieces) continue;
                        if (a.v_keep != nullptr)
                            *reinterpret_cast<uint4*>(reinterpret_cast<bf16*>(a.v_keep) + (size_t)t * a.ld_vk +
                                                      u * a.Dv + piece * 8) = pack8(v[c]);
                        if (a.v_first != nullptr) {
                            const float lam = a.lambda[0];
                            float f[8];
                            unpack8(*reinterpret_cast<const uint4*>(reinterpret_cast<const bf16*>(a.v_first) +
                                                                    (size_t)t * a.ld_vf + u * a.Dv + piece * 8), f);
#pragma unroll
                            for (int e = 0; e < 8; ++e) v[c][e] = (1.0f - lam) * v[c][e] + lam * f[e];
                        }
                    }
                }
            } else {
                if (ROW || kd.norm > 0) {
                    const float* nw = k == 0 ? a.q_norm_w : a.k_norm_w;
                    float r = k == 0 ? q_rstd : k_rstd;
                    if (!ROW) {
                        float ss = 0.f;
#pragma unroll
                        for (int c = 0; c < PIECES; ++c)
                            if (l + c * 32 < kd.norm) ss += square8(v[c]);
                        r = 1.0f / sqrtf(lanes_sum(ss, kd.shift) / (float)(kd.norm * 8) + a.eps);
                    }
                    const int normed = ROW ? kd.pieces : kd.norm;
#pragma unroll
                    for (int c = 0; c < PIECES; ++c) {
                        const int piece = l + c * 32;
                        if (u >= kd.units || piece >= normed) continue;
                        float w[8] = {1.f, 1.f, 1.f, 1.f, 1.f, 1.f, 1.f, 1.f};
                        if (nw != nullptr) load8_weights(nw + (ROW ? u * kd.stride : 0) + piece * 8, w);
#pragma unroll
                        for (int e = 0; e < 8; ++e) v[c][e] = v[c][e] * r * w[e];
                    }
                }
                if (a.rot_dims > 0) {
                    if (a.rot_half) {                     // (one piece a lane)
                        const int half = a.rot_dims >> 4, rel = l - kd.rot;
                        const bool low = rel >= 0 && rel < half, high = rel >= half && rel < 2 * half;
                        const int from = low ? lane + half : high ? lane - half : lane;
                        const int at = (low ? rel : high ? rel - half : 0) * 8;
#pragma unroll
                        for (int q = 0; q < 2; ++q) {
                            const float4 cs = *reinterpret_cast<const float4*>(cs_tab + at + 4 * q);
                            const float4 sn = *reinterpret_cast<const float4*>(sn_tab + at + 4 * q);
                            const float cc[4] = {cs.x, cs.y, cs.z, cs.w}, ss[4] = {sn.x, sn.y, sn.z, sn.w};
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                float& x = v[0][4 * q + e];
                                const float other = __shfl_sync(0xffffffffu, x, from);
                                const float turned = low ? x * cc[e] - other * ss[e] : x * cc[e] + other * ss[e];
                                x = low || high ? turned : x;
                            }
                        }
                    } else {
#pragma unroll
                        for (int c = 0; c < PIECES; ++c) {
                            const int rel = l + c * 32 - kd.rot;
                            if (rel < 0 || rel >= a.rot_dims >> 3) continue;
                            const float4 cs = *reinterpret_cast<const float4*>(cs_tab + rel * 4);
                            const float4 sn = *reinterpret_cast<const float4*>(sn_tab + rel * 4);
                            const float cc[4] = {cs.x, cs.y, cs.z, cs.w}, ss[4] = {sn.x, sn.y, sn.z, sn.w};
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                const float x = v[c][2 * e], y = v[c][2 * e + 1];
                                v[c][2 * e] = x * cc[e] - y * ss[e];
                                v[c][2 * e + 1] = y * cc[e] + x * ss[e];
                            }
                        }
                    }
                }
                if (kd.unit > 0) {
                    float ss = 0.f;
#pragma unroll
                    for (int c = 0; c < PIECES; ++c)
                        if (l + c * 32 < kd.unit) ss += square8(v[c]);
                    const float r = 1.0f / sqrtf(lanes_sum(ss, kd.shift) / (float)(kd.unit * 8) + a.eps);
#pragma unroll
                    for (int c = 0; c < PIECES; ++c)
                        if (l + c * 32 < kd.unit) {
#pragma unroll
                            for (int e = 0; e < 8; ++e) v[c][e] *= r;
                        }
                }
            }
#pragma unroll
            for (int c = 0; c < PIECES; ++c) {
                const int piece = l + c * 32;
                if (dst != nullptr && piece >= kd.skip && piece < kd.pieces)
                    *reinterpret_cast<uint4*>(dst + (piece - kd.skip) * 8) = pack8(v[c]);
            }
        }
    }
}

static int max_of(int a, int b, int c) { return a > b ? (a > c ? a : c) : (b > c ? b : c); }
static bool pieces(const void* p) { return ((uintptr_t)p & 15) == 0; }

// What is not written and enters no sum is not read either (a latent attention's unrotated queries).
static int head_prep_drop(int norm, int unit, int rot_off, int skip) {
    return norm == 0 && unit == 0 && rot_off >= skip ? skip : 0;
}

// One kind of vector for the kernel in pieces; false: it does not take these sizes.
static bool head_prep_kind(HeadPrepKind* kd, int off, int D, int units, int norm, int rot_off, int rot_dims,
                           int unit, int skip, int rot_half) {
    *kd = HeadPrepKind{};
    if (units == 0) return true;
    const int drop = head_prep_drop(norm, unit, rot_off, skip);
    if ((off | D | norm | rot_off | rot_dims | unit | skip) & 7) return false;
    if (rot_half && (rot_dims & 15)) return false;
    kd->off = off + drop;
    kd->stride = D;
    kd->pieces = (D - drop) / 8;
    if (kd->pieces < 1 || kd->pieces > 64 || (rot_half && rot_dims && kd->pieces > 32)) return false;
    while ((1 << kd->shift) < kd->pieces && kd->shift < 5) ++kd->shift;
    kd->units = units;
    kd->items = (units + (32 >> kd->shift) - 1) >> (5 - kd->shift);
    kd->norm = norm / 8;
    kd->rot = (rot_off - drop) / 8;
    kd->unit = unit / 8;
    kd->skip = (skip - drop) / 8;
    return true;
}

// Whether the kernel in pieces takes these arguments (bfloat16), and how it works on them: sizes and
// offsets in multiples of 8 elements, rows and weights on 16-byte boundaries, vectors of at most 512
// (256 where halves turn with one another), a token's vectors in one block's registers where all
// heads of a row are normed together.  Steps too small for what it packs stay with the general kernel,
// which spreads them over more warps.  General kernel / this one, us at 1 / 32 / 128 tokens:
//   short vectors, several to a warp: 4 + 2 + 2 heads of 64, normed and rotated, 3.2, 3.3, 3.4 / 3.5, 3.6, 3.6; of 32
//   +15, +12, +12 %; 14 + 2 + 2 of 64 +13, +12, +3 %; 3 + 3 + 3 of 96 and 64 +3, 0, 0 %.  From some 3,200 vectors
//   on this one is ahead (4 + 2 + 2 of 64, 511 tokens: 5.3 / 4.0).
//   a long normed row in one block, at 1 / 32 / 64 tokens: 40 + 8 + 8 heads of 128 5.0, 5.4, 9.4 / 5.9, 5.9, 6.0;
//   16 + 4 + 4 4.1, 4.3, 4.6 / 4.4, 4.5, 4.5; 32 + 8 + 8 of 64 +12, +4, -6 %.  Rows of up to 8 warps' worth of
//   vectors: -5 % and less.
static bool head_prep_plan(const HeadPrepArgs& a, int num_tokens, HeadPrepPlan* p, int* warps) {
    const bool has_v = a.v_off >= 0 && a.G > 0;
    if (((a.ld | a.ldq | a.q_head_stride) & 7) || !pieces(a.proj) || !pieces(a.q_out) || !pieces(a.k_cache) ||
        !pieces(a.v_cache) || !pieces(a.q_norm_w) || !pieces(a.k_norm_w) || !pieces(a.q_bias) || !pieces(a.k_bias) ||
        !pieces(a.v_bias))
        return false;
    if (a.v_first != nullptr && ((a.ld_vf & 7) || !pieces(a.v_first))) return false;
    if (a.v_keep != nullptr && ((a.ld_vk & 7) || !pieces(a.v_keep))) return false;
    const int rd = a.rot_dims;
    if (a.row_norm && a.q_skip) return false;
    if (!head_prep_kind(&p->kind[0], a.q_off, a.Dq, a.H, a.row_norm ? 0 : a.q_norm_dims, rd ? a.q_rot_off : 0, rd,
                        a.q_unit_dims, a.q_skip, a.rot_half) ||
        !head_prep_kind(&p->kind[1], a.k_off, a.Dk, a.G, a.row_norm ? 0 : a.k_norm_dims, rd ? a.k_rot_off : 0, rd,
                        a.k_unit_dims, 0, a.rot_half) ||
        !head_prep_kind(&p->kind[2], a.v_off, a.Dv, has_v ? a.G : 0, 0, 0, 0, 0, 0, 0))
        return false;
    p->items = p->kind[0].items + p->kind[1].items + p->kind[2].items;
    const int units = a.H + a.G + (has_v ? a.G : 0), longest = max_of(a.Dq, a.Dk, has_v ? a.Dv : 0);
    if (a.row_norm ? num_tokens <= 32 && p->items > 8 : longest <= 96 && (long long)num_tokens * units <= 3200)
        return false;
    *warps = a.row_norm && (p->items > 4 * HPV_ITEMS || num_tokens < 512) ? 8 : 4;
    return !a.row_norm || p->items <= *warps * HPV_ITEMS;
}

// out = x * sigmoid(gate), float32 arithmetic; one gate value per `group` neighbouring elements
// (1: element by element; a head's size: one number a head).
template <typename T>
__global__ void __launch_bounds__(256) sigmoid_gate_kernel(const T* __restrict__ x, int ldx,
                                                           const T* __restrict__ gate, int ldg,
                                                           T* __restrict__ out, int ldo, int N, int group) {
    pdl_wait();
    pdl_launch_dependents();
    const size_t t = blockIdx.x;
    for (int c = threadIdx.x; c < N; c += blockDim.x) {
        const float z = to_float(gate[t * ldg + c / group]);
        const float v = to_float(x[t * ldx + c]);
        out[t * ldo + c] = from_float<T>(sizeof(T) == 2 ? v * sigmoid_for<T>(z) : v / (1.0f + expf(-z)));
    }
}

// The same on bfloat16 rows in 16-byte pieces (8 elements under one gate value or 8 of them): a piece a
// thread over all rows, so that every load is in flight at once (2,082 rows of 2,048: 14.6 -> 7.0 us; 2,048
// rows 5.7 -> 4.4 with the approximate reciprocal).
__global__ void __launch_bounds__(256) sigmoid_gate_vec_kernel(const bf16* __restrict__ x, int ldx,
                                                               const bf16* __restrict__ gate, int ldg,
                                                               bf16* __restrict__ out, int ldo, int row_pieces,
                                                               int group, long long total) {
    pdl_wait();
    pdl_launch_dependents();
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
    if (i >= total) return;
    const long long t = i / row_pieces;
    const int c = (int)(i - t * row_pieces) * 8;
    float v[8], z[8];
    const uint4 raw = *reinterpret_cast<const uint4*>(x + t * ldx + c);
    if (group == 1) {
        unpack8(*reinterpret_cast<const uint4*>(gate + t * ldg + c), z);
    } else {
        const float g = to_float(gate[t * ldg + c / group]);
#pragma unroll
        for (int e = 0; e < 8; ++e) z[e] = g;
    }
    unpack8(raw, v);
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] *= sigmoid_for<bf16>(z[e]);
    *reinterpret_cast<uint4*>(out + t * ldo + c) = pack8(v);
}

template <typename T>
static int launch_head_prep(const HeadPrepArgs& a, int num_tokens, cudaStream_t st) {
    if (num_tokens <= 0) return 0;
    const int maxd = max_of(a.Dq, a.Dk, a.Dv);
    if (a.H < 0 || a.G < 0 || a.Dq < 0 || a.Dk < 0 || maxd <= 0 || (a.rot_dims & 1)) return SLB_ERR_BAD_ARG;
    if (maxd > HP_MAX_D) return SLB_ERR_TOO_LARGE;
    if (a.rot_dims > 0 && (a.freq == nullptr || (a.H > 0 && a.q_rot_off + a.rot_dims > a.Dq) ||
                           (a.G > 0 && a.k_rot_off + a.rot_dims > a.Dk)))
        return SLB_ERR_BAD_ARG;
    if (a.row_norm && (a.q_norm_w == nullptr || a.k_norm_w == nullptr || a.H <= 0 || a.G <= 0)) return SLB_ERR_BAD_ARG;
    if (a.q_norm_dims > a.Dq || a.k_norm_dims > a.Dk || a.q_skip < 0 || a.q_skip > a.Dq) return SLB_ERR_BAD_ARG;
    if (a.q_unit_dims < 0 || a.q_unit_dims > a.Dq || a.k_unit_dims < 0 || a.k_unit_dims > a.Dk) return SLB_ERR_BAD_ARG;
    if ((a.k_cache != nullptr || a.v_cache != nullptr) && (a.block_table == nullptr || a.page_size <= 0))
        return SLB_ERR_BAD_ARG;
    HeadPrepPlan plan;
    int warps;
    if (sizeof(T) == 2 && head_prep_plan(a, num_tokens, &plan, &warps)) {
        // (a step of few tokens: a block a few vectors, so that it still fills the device)
        const int split = num_tokens < 512 && !a.row_norm ? (plan.items + warps - 1) / warps : 1;
        const bool wide = plan.kind[0].pieces > 32 || plan.kind[1].pieces > 32 || plan.kind[2].pieces > 32;
        auto pick = [&](auto dense) {
            return a.row_norm ? (wide ? head_prep_vec_kernel<2, true, dense.value> : head_prep_vec_kernel<1, true, dense.value>)
                              : (wide ? head_prep_vec_kernel<2, false, dense.value> : head_prep_vec_kernel<1, false, dense.value>);
        };
        // (a block is a chain of latencies, 2.8 us, and a round of blocks costs that whatever it holds: with more warps an
        // SM, spilled registers and an eighth (long vectors: a third) more a round, when that saves rounds.  16 + 4 heads
        // of 128 turned: 1,024 tokens 9.8 -> 8.0 us, 2,048 14.4 -> 12.7; 40 + 8 heads 1,024 22.7 -> 16.9; all steps with
        // it: 700 tokens 1.2-1.3 times as long, 256 the same)
        const long long blocks = (long long)num_tokens * split, sms = slb_num_sms();
        const long long usual = sms * ((wide ? 16 : 24) / warps), dense = sms * ((wide ? 24 : 32) / warps);
        const bool fewer = 24 * ((blocks + usual - 1) / usual) > (wide ? 32 : 27) * ((blocks + dense - 1) / dense);
        auto kernel = fewer ? pick(std::true_type{}) : pick(std::false_type{});
        HeadPrepArgs read = a;                           // (a bias has the elements too that are not read)
        if (a.q_bias != nullptr && !a.row_norm)
            read.q_bias += head_prep_drop(a.q_norm_dims, a.q_unit_dims, a.rot_dims ? a.q_rot_off : 0, a.q_skip);
        return slb_launch(kernel, dim3(num_tokens, split), dim3(warps * 32), a.rot_dims * sizeof(float), st, read, plan);
    }
    const size_t smem = ((size_t)HP_WARPS * maxd + a.rot_dims) * sizeof(float);
    const int units = a.H + a.G + (a.v_off >= 0 ? a.G : 0);
    const int gy = num_tokens < 512 ? (units + HP_WARPS - 1) / HP_WARPS : 1;
    return slb_launch(head_prep_kernel<T>, dim3(num_tokens, gy), dim3(HP_WARPS * 32), smem, st, a);
}

extern "C" {
int slb_head_prep_f32(const HeadPrepArgs* a, int num_tokens, cudaStream_t st) {
    return launch_head_prep<float>(*a, num_tokens, st);
}
int slb_head_prep_bf16(const HeadPrepArgs* a, int num_tokens, cudaStream_t st) {
    return launch_head_prep<bf16>(*a, num_tokens, st);
}
int slb_sigmoid_gate_f32(const float* x, int ldx, const float* gate, int ldg, float* out, int ldo, int T,
                         int N, int group, cudaStream_t st) {
    if (T <= 0 || N <= 0) return 0;
    if (group <= 0) return SLB_ERR_BAD_ARG;
    return slb_launch(sigmoid_gate_kernel<float>, dim3(T), dim3(256), 0, st, x, ldx, gate, ldg, out, ldo, N, group);
}
int slb_sigmoid_gate_bf16(const bf16* x, int ldx, const bf16* gate, int ldg, bf16* out, int ldo, int T,
                          int N, int group, cudaStream_t st) {
    if (T <= 0 || N <= 0) return 0;
    if (group <= 0) return SLB_ERR_BAD_ARG;
    if (((ldx | ldo | N) & 7) == 0 && pieces(x) && pieces(out) &&
        (group == 1 ? (ldg & 7) == 0 && pieces(gate) : (group & 7) == 0)) {
        const long long total = (long long)T * (N / 8), blocks = (total + 255) / 256;
        if (blocks <= 0x7fffffffll)
            return slb_launch(sigmoid_gate_vec_kernel, dim3((unsigned)blocks), dim3(256), 0, st, x, ldx, gate, ldg, out,
                              ldo, N / 8, group, total);
    }
    return slb_launch(sigmoid_gate_kernel<bf16>, dim3(T), dim3(256), 0, st, x, ldx, gate, ldg, out, ldo, N, group);
}
}

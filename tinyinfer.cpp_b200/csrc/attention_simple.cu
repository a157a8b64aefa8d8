// Attention on the CUDA cores, for every head size and both cache types.
//
//  * qk_norm_rope_store: per-head RMSNorm of q and k, NeoX rotation at the token's position,
//    k and v written once per kv head into the token's page, q written for the attention kernel.
//  * paged_attention_simple: one block per (token, query head); its warps share the keys of the
//    token's context [lo, pos] (lo > 0 only for a window) and merge their online softmaxes.
//
// These are the true 32-bit kernels and the fallback of the bfloat16 path for shapes that
// the tensor-core kernels refuse.  Cache layout: pages[page][0 = keys, 1 = values][kv head]
// [slot][head_dim]; a token at position p of request r lies in page block_table[r][p / page_size],
// slot p % page_size.
#include "common.cuh"
#include "tape.cuh"

namespace {

constexpr int MAX_HEAD_DIM = 256;
constexpr int WARPS = 4;

enum { TI_ERR_BAD_PAGE = 1 };
template <int N> struct Int { static constexpr int value = N; };

template <typename TQ, typename TC>
__global__ void __launch_bounds__(WARPS * 32)
qk_norm_rope_store_kernel(const float* qkv, int qkv_stride,
                          const float* __restrict__ q_weight, const float* __restrict__ k_weight,
                          float eps, const float* __restrict__ inv_freq,
                          const int* __restrict__ positions, const int* __restrict__ req_of_tok,
                          const int* __restrict__ block_table, int bt_stride,
                          TC* __restrict__ pages, int num_pages, int page_size, int write_kv,
                          int num_heads, int num_kv_heads, int head_dim, int rotary_dim,
                          TQ* __restrict__ q_out, int* __restrict__ status) {
    __shared__ float vec[WARPS][MAX_HEAD_DIM];
    pdl_launch();
    pdl_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t = blockIdx.x;
    const int item = blockIdx.y * WARPS + warp;
    const int items = num_heads + 2 * num_kv_heads;
    if (item >= items) return;
    const int half = rotary_dim >> 1;                 // pairs (k, k + half), k < half, are rotated
    const int nq = num_heads * head_dim, nk = num_kv_heads * head_dim;
    const int pos = positions[t];

    // which vector: a query head, a key head or a value head
    int kind, head;
    if (item < num_heads) { kind = 0; head = item; }
    else if (item < num_heads + num_kv_heads) { kind = 1; head = item - num_heads; }
    else { kind = 2; head = item - num_heads - num_kv_heads; }
    if (kind != 0 && !write_kv) return;
    const float* src = qkv + (size_t)t * qkv_stride +
                       (kind == 0 ? head * head_dim : kind == 1 ? nq + head * head_dim
                                                                : nq + nk + head * head_dim);
    TC* dst = nullptr;
    if (kind != 0) {
        const int r = req_of_tok[t];
        const int page = block_table[(size_t)r * bt_stride + pos / page_size];
        if (page < 0 || page >= num_pages) {
            if (lane == 0) atomicCAS(status, 0, TI_ERR_BAD_PAGE);
            return;
        }
        dst = pages + ((((size_t)page * 2 + (kind - 1)) * num_kv_heads + head) * page_size +
                       pos % page_size) * head_dim;
    }
    if (kind == 2) {                                   // values are stored as they are
        for (int d = lane; d < head_dim; d += 32) dst[d] = from_f32<TC>(src[d]);
        return;
    }
    const float* w = kind == 0 ? q_weight : k_weight;
    float ss = 0.0f;
    for (int d = lane; d < head_dim; d += 32) {
        const float v = src[d];
        vec[warp][d] = v;
        ss = fmaf(v, v, ss);
    }
    ss = warp_sum(ss);
    const float inv = 1.0f / sqrtf(ss / (float)head_dim + eps);
    __syncwarp();
    for (int k = lane; k < half; k += 32) {
        const float x0 = vec[warp][k] * inv * w[k];
        const float x1 = vec[warp][k + half] * inv * w[k + half];
        const float angle = (float)pos * inv_freq[k];
        float sn, cs;
        sincosf(angle, &sn, &cs);
        const float y0 = x0 * cs - x1 * sn;
        const float y1 = x0 * sn + x1 * cs;
        if (kind == 0) {
            TQ* q = q_out + (size_t)t * nq + head * head_dim;
            q[k] = from_f32<TQ>(y0);
            q[k + half] = from_f32<TQ>(y1);
        } else {
            dst[k] = from_f32<TC>(y0);
            dst[k + half] = from_f32<TC>(y1);
        }
    }
    // what lies beyond the rotated width is normed only
    for (int d = rotary_dim + lane; d < head_dim; d += 32) {
        const float y = vec[warp][d] * inv * w[d];
        if (kind == 0) q_out[(size_t)t * nq + head * head_dim + d] = from_f32<TQ>(y);
        else dst[d] = from_f32<TC>(y);
    }
}

// The same work for head sizes up to 64 * VEC with head_dim / 2 a multiple of VEC: a lane keeps
// VEC consecutive elements of each half of the vector in registers (the rotation pairs element
// k with k + head_dim / 2, so a lane owns whole pairs); no shared memory.
template <typename TQ, typename TC, int VEC>
__global__ void __launch_bounds__(WARPS * 32)
qk_norm_rope_store_vec_kernel(const float* qkv, int qkv_stride,
                              const float* __restrict__ q_weight, const float* __restrict__ k_weight,
                              float eps, const float* __restrict__ inv_freq,
                              const int* __restrict__ positions, const int* __restrict__ req_of_tok,
                              const int* __restrict__ block_table, int bt_stride,
                              TC* __restrict__ pages, int num_pages, int page_size, int write_kv,
                              int num_heads, int num_kv_heads, int head_dim, int items_per_warp,
                              TQ* __restrict__ q_out, int* __restrict__ status) {
    __shared__ float cs_tab[MAX_HEAD_DIM / 2], sn_tab[MAX_HEAD_DIM / 2];
    pdl_launch();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t = blockIdx.x;
    const int half = head_dim >> 1;
    const int nq = num_heads * head_dim, nk = num_kv_heads * head_dim;
    const int pos = positions[t];
    // the rotation of a token is the same for all its heads: its sines and cosines once per block
    for (int k = threadIdx.x; k < half; k += WARPS * 32)
        sincosf((float)pos * inv_freq[k], &sn_tab[k], &cs_tab[k]);
    pdl_wait();
    __syncthreads();
    // With many tokens a warp takes up to MAX_TURNS vectors, so that blocks are not tiny; all of
    // their loads are issued before any of them is used.  (Few tokens take
    // qk_norm_rope_store_one_kernel below.)
    constexpr int MAX_TURNS = 8;
    const int items = num_heads + 2 * num_kv_heads;
    const int k0 = lane * VEC;
    const bool active = k0 < half;
    float lo[MAX_TURNS][VEC], hi[MAX_TURNS][VEC];
#pragma unroll
    for (int turn = 0; turn < MAX_TURNS; ++turn) {
        const int item = (blockIdx.y * items_per_warp + turn) * WARPS + warp;
        const bool live = turn < items_per_warp && item < items && active;
        const float* src = qkv + (size_t)t * qkv_stride + (size_t)(live ? item : 0) * head_dim;
#pragma unroll
        for (int i = 0; i < VEC; ++i) {
            lo[turn][i] = live ? src[k0 + i] : 0.0f;
            hi[turn][i] = live ? src[half + k0 + i] : 0.0f;
        }
    }
    int page = -1;
    if (write_kv) {
        page = block_table[(size_t)req_of_tok[t] * bt_stride + pos / page_size];
        if (page < 0 || page >= num_pages) {
            if (threadIdx.x == 0) atomicCAS(status, 0, TI_ERR_BAD_PAGE);
            page = -1;
        }
    }
#pragma unroll
    for (int turn = 0; turn < MAX_TURNS; ++turn) {
        const int item = (blockIdx.y * items_per_warp + turn) * WARPS + warp;
        if (turn >= items_per_warp || item >= items) break;
        // the vectors of a token lie one after the other: query heads, key heads, value heads
        const int kind = item < num_heads ? 0 : item < num_heads + num_kv_heads ? 1 : 2;
        const int head = kind == 0 ? item : kind == 1 ? item - num_heads : item - num_heads - num_kv_heads;
        if (kind != 0 && page < 0) continue;
        TC* dst = nullptr;
        if (kind != 0)
            dst = pages + ((((size_t)page * 2 + (kind - 1)) * num_kv_heads + head) * page_size +
                           pos % page_size) * head_dim;
        if (kind == 2) {
            if (active) {
#pragma unroll
                for (int i = 0; i < VEC; ++i) {
                    dst[k0 + i] = from_f32<TC>(lo[turn][i]);
                    dst[half + k0 + i] = from_f32<TC>(hi[turn][i]);
                }
            }
            continue;
        }
        float ss = 0.0f;
#pragma unroll
        for (int i = 0; i < VEC; ++i) {
            ss = fmaf(lo[turn][i], lo[turn][i], ss);
            ss = fmaf(hi[turn][i], hi[turn][i], ss);
        }
        ss = warp_sum(ss);
        const float inv = 1.0f / sqrtf(ss / (float)head_dim + eps);
        if (!active) continue;
        const float* w = kind == 0 ? q_weight : k_weight;
#pragma unroll
        for (int i = 0; i < VEC; ++i) {
            const float x0 = lo[turn][i] * inv * w[k0 + i];
            const float x1 = hi[turn][i] * inv * w[half + k0 + i];
            const float sn = sn_tab[k0 + i], cs = cs_tab[k0 + i];
            const float y0 = x0 * cs - x1 * sn;
            const float y1 = x0 * sn + x1 * cs;
            if (kind == 0) {
                TQ* q = q_out + (size_t)t * nq + head * head_dim;
                q[k0 + i] = from_f32<TQ>(y0);
                q[half + k0 + i] = from_f32<TQ>(y1);
            } else {
                dst[k0 + i] = from_f32<TC>(y0);
                dst[half + k0 + i] = from_f32<TC>(y1);
            }
        }
    }
}

// The same work for the few tokens of a decode step, one vector per warp: everything that does
// not come from the kernel before (the token's position and page, its sines and cosines, the norm
// weights) is in registers before the wait for that kernel returns, so that behind the wait
// there is one round of loads, the norm, the rotation and the stores.  Arithmetic and order are
// those of qk_norm_rope_store_vec_kernel.
template <typename TQ, typename TC, int VEC>
__global__ void __launch_bounds__(WARPS * 32)
qk_norm_rope_store_one_kernel(const float* qkv, int qkv_stride,
                              const float* __restrict__ q_weight, const float* __restrict__ k_weight,
                              float eps, const float* __restrict__ inv_freq,
                              const int* __restrict__ positions, const int* __restrict__ req_of_tok,
                              const int* __restrict__ block_table, int bt_stride,
                              TC* __restrict__ pages, int num_pages, int page_size, int write_kv,
                              int num_heads, int num_kv_heads, int head_dim,
                              TQ* __restrict__ q_out, int* __restrict__ status) {
    pdl_launch();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t = blockIdx.x;
    const int half = head_dim >> 1;
    const int items = num_heads + 2 * num_kv_heads;
    const int item = blockIdx.y * WARPS + warp;
    const int k0 = lane * VEC;
    const bool active = k0 < half, live = item < items;
    // the vectors of a token lie one after the other: query heads, key heads, value heads
    const int kind = item < num_heads ? 0 : item < num_heads + num_kv_heads ? 1 : 2;
    const int head = kind == 0 ? item : kind == 1 ? item - num_heads : item - num_heads - num_kv_heads;
    const int pos = positions[t];
    int page = -1;
    if (write_kv && kind != 0 && live) {
        page = block_table[(size_t)req_of_tok[t] * bt_stride + pos / page_size];
        if (page < 0 || page >= num_pages) {
            if (lane == 0) atomicCAS(status, 0, TI_ERR_BAD_PAGE);
            page = -1;
        }
    }
    float sn[VEC], cs[VEC], w0[VEC], w1[VEC];
    if (live && active && kind != 2) {
        const float* w = kind == 0 ? q_weight : k_weight;
#pragma unroll
        for (int i = 0; i < VEC; ++i) {
            sincosf((float)pos * inv_freq[k0 + i], &sn[i], &cs[i]);
            w0[i] = w[k0 + i];
            w1[i] = w[half + k0 + i];
        }
    }
    pdl_wait();
    if (!live) return;
    float lo[VEC], hi[VEC];
    const float* src = qkv + (size_t)t * qkv_stride + (size_t)item * head_dim;
#pragma unroll
    for (int i = 0; i < VEC; ++i) {
        lo[i] = active ? src[k0 + i] : 0.0f;
        hi[i] = active ? src[half + k0 + i] : 0.0f;
    }
    if (kind != 0 && page < 0) return;
    TC* dst = nullptr;
    if (kind != 0)
        dst = pages + ((((size_t)page * 2 + (kind - 1)) * num_kv_heads + head) * page_size +
                       pos % page_size) * head_dim;
    if (kind == 2) {
        if (active) {
#pragma unroll
            for (int i = 0; i < VEC; ++i) {
                dst[k0 + i] = from_f32<TC>(lo[i]);
                dst[half + k0 + i] = from_f32<TC>(hi[i]);
            }
        }
        return;
    }
    float ss = 0.0f;
#pragma unroll
    for (int i = 0; i < VEC; ++i) {
        ss = fmaf(lo[i], lo[i], ss);
        ss = fmaf(hi[i], hi[i], ss);
    }
    ss = warp_sum(ss);
    const float inv = 1.0f / sqrtf(ss / (float)head_dim + eps);
    if (!active) return;
#pragma unroll
    for (int i = 0; i < VEC; ++i) {
        const float x0 = lo[i] * inv * w0[i];
        const float x1 = hi[i] * inv * w1[i];
        const float y0 = x0 * cs[i] - x1 * sn[i];
        const float y1 = x0 * sn[i] + x1 * cs[i];
        if (kind == 0) {
            TQ* q = q_out + ((size_t)t * num_heads + head) * head_dim;
            q[k0 + i] = from_f32<TQ>(y0);
            q[half + k0 + i] = from_f32<TQ>(y1);
        } else {
            dst[k0 + i] = from_f32<TC>(y0);
            dst[half + k0 + i] = from_f32<TC>(y1);
        }
    }
}

// One block per (token, query head).  The warps take the keys of [lo, pos] in turn (key lo + w, lo + w +
// ATT_WARPS, ...), each with an online softmax of its own, merged at the end: an order that depends on the row
// alone.  A warp's time is the latency of its loads and of the sum over its lanes, so it asks for the keys and
// values of AHEAD keys at once and adds their dot products side by side; the online softmax then takes them one
// after the other (so AHEAD changes no bit), and fewer keys than that are taken in halves.  PER_LANE elements of a head
// per lane.  Keys asked for ahead cost registers and so blocks on an SM: many blocks cover one another's latency and take
// one key at a time (see the launch).
constexpr int ATT_WARPS = 8;

template <typename TQ, typename TC, int PER_LANE, int AHEAD>
__global__ void __launch_bounds__(ATT_WARPS * 32, AHEAD > 1 ? 1 : PER_LANE <= 4 ? 8 : 4)
paged_attention_simple_kernel(const TQ* q, const int* __restrict__ rows, const int* __restrict__ positions,
                              const int* __restrict__ req_of_tok, const int* __restrict__ block_table, int bt_stride,
                              const TC* pages, int num_pages, int page_size, int num_heads, int num_kv_heads,
                              int head_dim, int window, float scale, TQ* out, int* __restrict__ status) {
    __shared__ float so[ATT_WARPS][32 * PER_LANE];
    __shared__ float sm[ATT_WARPS], sl[ATT_WARPS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int h = blockIdx.y, t = rows ? rows[blockIdx.x] : blockIdx.x;
    const int kvh = h / (num_heads / num_kv_heads);
    const int pos = positions[t];
    const int r = req_of_tok[t];
    const int lo = window > 0 ? max(0, pos - window + 1) : 0;
    const int* table = block_table + (size_t)r * bt_stride;
    pdl_launch();
    pdl_wait();

    float qv[PER_LANE], o[PER_LANE];
    const TQ* qh = q + ((size_t)t * num_heads + h) * head_dim;
#pragma unroll
    for (int i = 0; i < PER_LANE; ++i) {
        const int d = lane + 32 * i;
        qv[i] = d < head_dim ? to_f32(qh[d]) : 0.0f;
        o[i] = 0.0f;
    }
    float m = -INFINITY, l = 0.0f;
    bool bad = false;
    const size_t to_values = (size_t)num_kv_heads * page_size * head_dim;
    // N keys, ATT_WARPS apart, of which the last is no later than pos
    auto take = [&](int p0, auto n) {
        constexpr int N = decltype(n)::value;
        TC kv[N][PER_LANE], vv[N][PER_LANE];
        bool there[N];
#pragma unroll
        for (int j = 0; j < N; ++j) {
            const int p = p0 + j * ATT_WARPS;
            const int page = table[p / page_size];
            there[j] = page >= 0 && page < num_pages;
            bad |= !there[j];
            const TC* kp = pages + (((size_t)page * 2 * num_kv_heads + kvh) * page_size + p % page_size) * head_dim;
#pragma unroll
            for (int i = 0; i < PER_LANE; ++i) {
                const int d = lane + 32 * i;
                const bool on = there[j] && d < head_dim;
                kv[j][i] = on ? kp[d] : from_f32<TC>(0.0f);
                vv[j][i] = on ? kp[to_values + d] : from_f32<TC>(0.0f);
            }
        }
        float s[N];
#pragma unroll
        for (int j = 0; j < N; ++j) {
            s[j] = 0.0f;
#pragma unroll
            for (int i = 0; i < PER_LANE; ++i) s[j] = fmaf(qv[i], to_f32(kv[j][i]), s[j]);
        }
#pragma unroll
        for (int x = 16; x > 0; x >>= 1)
#pragma unroll
            for (int j = 0; j < N; ++j) s[j] += __shfl_xor_sync(0xffffffffu, s[j], x);
#pragma unroll
        for (int j = 0; j < N; ++j) {
            if (!there[j]) continue;
            const float sc = s[j] * scale;
            const float m_new = fmaxf(m, sc);
            const float alpha = expf(m - m_new);          // exp(-inf) = 0 on the first key
            const float pr = expf(sc - m_new);
            l = l * alpha + pr;
#pragma unroll
            for (int i = 0; i < PER_LANE; ++i) o[i] = fmaf(pr, to_f32(vv[j][i]), o[i] * alpha);
            m = m_new;
        }
    };
    int p = lo + warp;
    for (; p + (AHEAD - 1) * ATT_WARPS <= pos; p += AHEAD * ATT_WARPS) take(p, Int<AHEAD>{});
    if (AHEAD > 4 && p + 3 * ATT_WARPS <= pos) { take(p, Int<4>{}); p += 4 * ATT_WARPS; }
    if (AHEAD > 2 && p + ATT_WARPS <= pos) { take(p, Int<2>{}); p += 2 * ATT_WARPS; }
    if (p <= pos) take(p, Int<1>{});
    if (bad && lane == 0) atomicCAS(status, 0, TI_ERR_BAD_PAGE);
#pragma unroll
    for (int i = 0; i < PER_LANE; ++i) so[warp][lane + 32 * i] = o[i];
    if (lane == 0) { sm[warp] = m; sl[warp] = l; }
    __syncthreads();
    if (threadIdx.x >= 32 * PER_LANE) return;
    float mm = -INFINITY;
#pragma unroll
    for (int w = 0; w < ATT_WARPS; ++w) mm = fmaxf(mm, sm[w]);
    float ltot = 0.0f, wt[ATT_WARPS];
#pragma unroll
    for (int w = 0; w < ATT_WARPS; ++w) {
        wt[w] = sl[w] > 0.0f ? expf(sm[w] - mm) : 0.0f;
        ltot += sl[w] * wt[w];
    }
    const float inv = 1.0f / ltot;
    TQ* oh = out + ((size_t)t * num_heads + h) * head_dim;
    if (threadIdx.x < head_dim) {
        const int d = threadIdx.x;
        float acc = 0.0f;
#pragma unroll
        for (int w = 0; w < ATT_WARPS; ++w) acc = fmaf(so[w][d], wt[w], acc);
        oh[d] = from_f32<TQ>(acc * inv);
    }
}

// The same for up to ROWS consecutive tokens of one request a block (no window): a key and its value are read once for all of
// them, which is what bounds many rows (466 tokens of three prompts, 16 heads of 128: 600 MB from L2, 122 us a layer -> 65).
// A row takes the same keys in the same order through the same arithmetic as above, so its bits are those of the kernel above:
// the sums over the lanes are the same tree, folded for all rows at once (a lane is left with the score of row lane / 4, whose
// maximum, sum and exponentials it keeps and hands out).  All ROWS scores are made for every key, so rows of different
// requests gain nothing from one block: 80 single tokens at 1,000 keys walked eight to a block 810 us, by the kernel above 244.
// tiles[i] = {request row, first flat token, tokens}, of at most runs * ROWS tokens.  The grid has the heads of a run beside one
// another and a tile's last tokens first, so that the blocks with the most keys come first (466 tokens of three prompts 52 to
// 61 us; a tile of 64 tokens with its runs last in the grid 73).
constexpr int ROWS = 8, ROW_LANES = 32 / ROWS;

template <typename TQ, typename TC, int PER_LANE>
__global__ void __launch_bounds__(ATT_WARPS * 32, PER_LANE <= 4 ? 2 : 1)
paged_attention_rows_kernel(const TQ* q, const int* __restrict__ tiles, int runs, const int* __restrict__ positions,
                            const int* __restrict__ block_table, int bt_stride, const TC* pages, int num_pages, int page_size,
                            int num_heads, int num_kv_heads, int head_dim, float scale, TQ* out, int* __restrict__ status) {
    __shared__ float so[ATT_WARPS][ROWS / 2][32 * PER_LANE];
    __shared__ float sm[ATT_WARPS][ROWS], sl[ATT_WARPS][ROWS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int run = blockIdx.x / num_heads, h = blockIdx.x - run * num_heads;
    const int* tile = tiles + 3 * (run / runs);
    const int first = ROWS * (runs - 1 - run % runs), t0 = tile[1] + first;
    const int count = min(ROWS, tile[2] - first);
    if (count <= 0) return;
    const int kvh = h / (num_heads / num_kv_heads);
    pdl_launch();
    pdl_wait();
    const size_t to_values = (size_t)num_kv_heads * page_size * head_dim;
    bool bad = false;
    const int* table = block_table + (size_t)tile[0] * bt_stride;
    const int own = lane / ROW_LANES;                        // this lane's row
    int pos[ROWS], last = 0, least = 1 << 30;
    float qv[ROWS][PER_LANE], o[ROWS][PER_LANE];
#pragma unroll
    for (int j = 0; j < ROWS; ++j) {
        const int t = t0 + j;
        pos[j] = j < count ? positions[t] : -1;
        last = max(last, pos[j]);
        least = j < count ? min(least, pos[j]) : least;
#pragma unroll
        for (int i = 0; i < PER_LANE; ++i) {
            const int d = lane + 32 * i;
            qv[j][i] = j < count && d < head_dim ? to_f32(q[((size_t)t * num_heads + h) * head_dim + d]) : 0.0f;
            o[j][i] = 0.0f;
        }
    }
    int my_pos = -1;
#pragma unroll
    for (int j = 0; j < ROWS; ++j) my_pos = own == j ? pos[j] : my_pos;
    float m = -INFINITY, l = 0.0f;                   // of row `own`
    constexpr int DEEP = 2;                          // keys of this warp on their way
    TC kn[DEEP][PER_LANE], vn[DEEP][PER_LANE];
    bool there_next[DEEP];
    // the keys of a warp follow one another: the page is looked up where it changes, and nothing is divided
    int block = warp / page_size, slot = warp - block * page_size, page = -1;
    const TC* base = pages;
    auto turn_page = [&]() {
        page = block * page_size <= last ? table[block] : -1;
        base = pages + ((size_t)(page >= 0 && page < num_pages ? page : 0) * 2 * num_kv_heads + kvh) * page_size * head_dim;
    };
    turn_page();
    auto fetch = [&](int p, TC (&kn)[PER_LANE], TC (&vn)[PER_LANE], bool& there) {
        if (p > last) return;
        there = page >= 0 && page < num_pages;
        const TC* kp = base + (size_t)slot * head_dim;
#pragma unroll
        for (int i = 0; i < PER_LANE; ++i) {
            const int d = lane + 32 * i;
            const bool on = there && d < head_dim;
            kn[i] = on ? kp[d] : from_f32<TC>(0.0f);
            vn[i] = on ? kp[to_values + d] : from_f32<TC>(0.0f);
        }
        slot += ATT_WARPS;
        if (slot >= page_size) {
            do { slot -= page_size; ++block; } while (slot >= page_size);
            turn_page();
        }
    };
    auto take = [&](int p, TC (&kn)[PER_LANE], TC (&vn)[PER_LANE], bool& there_then) {
        float kf[PER_LANE], vf[PER_LANE];
#pragma unroll
        for (int i = 0; i < PER_LANE; ++i) { kf[i] = to_f32(kn[i]); vf[i] = to_f32(vn[i]); }
        const bool there = there_then;
        fetch(p + DEEP * ATT_WARPS, kn, vn, there_then);
        if (!there) { bad = true; return; }
        float s[ROWS];
#pragma unroll
        for (int j = 0; j < ROWS; ++j) {
            s[j] = 0.0f;
#pragma unroll
            for (int i = 0; i < PER_LANE; ++i) s[j] = fmaf(qv[j][i], kf[i], s[j]);
        }
        // sums over the lanes: a lane keeps half of its rows at each exchange until it has one
#pragma unroll
        for (int half = ROWS / 2, x = 16; half >= 1; half >>= 1, x >>= 1) {
            const bool upper = lane & x;
#pragma unroll
            for (int j = 0; j < half; ++j) {
                const float keep = upper ? s[j + half] : s[j], give = upper ? s[j] : s[j + half];
                s[j] = keep + __shfl_xor_sync(0xffffffffu, give, x);
            }
        }
#pragma unroll
        for (int x = ROW_LANES / 2; x >= 1; x >>= 1) s[0] += __shfl_xor_sync(0xffffffffu, s[0], x);
        float alpha = 1.0f, pr = 0.0f;
        const bool sees = p <= my_pos;
        if (sees) {
            const float sc = s[0] * scale, m_new = fmaxf(m, sc);
            alpha = expf(m - m_new);                 // exp(-inf) = 0 on the first key
            pr = expf(sc - m_new);
            l = l * alpha + pr;
            m = m_new;
        }
        if (p <= least && !__any_sync(0xffffffffu, alpha != 1.0f)) {     // every row sees it, no maximum moved
#pragma unroll
            for (int j = 0; j < ROWS; ++j) {
                const float w = __shfl_sync(0xffffffffu, pr, ROW_LANES * j);
#pragma unroll
                for (int i = 0; i < PER_LANE; ++i) o[j][i] = fmaf(w, vf[i], o[j][i]);
            }
            return;
        }
#pragma unroll
        for (int j = 0; j < ROWS; ++j) {
            const float a = __shfl_sync(0xffffffffu, alpha, ROW_LANES * j), w = __shfl_sync(0xffffffffu, pr, ROW_LANES * j);
            if (p > pos[j]) continue;
#pragma unroll
            for (int i = 0; i < PER_LANE; ++i) o[j][i] = fmaf(w, vf[i], o[j][i] * a);
        }
    };
#pragma unroll
    for (int d = 0; d < DEEP; ++d) fetch(warp + d * ATT_WARPS, kn[d], vn[d], there_next[d]);
    for (int p = warp; p <= last; p += DEEP * ATT_WARPS) {
#pragma unroll
        for (int d = 0; d < DEEP; ++d)
            if (p + d * ATT_WARPS <= last) take(p + d * ATT_WARPS, kn[d], vn[d], there_next[d]);
    }
    if (lane % ROW_LANES == 0) { sm[warp][own] = m; sl[warp][own] = l; }
#pragma unroll
    for (int part = 0; part < 2; ++part) {           // half of the rows at a time meet in shared memory
        __syncthreads();
#pragma unroll
        for (int j = 0; j < ROWS / 2; ++j)
#pragma unroll
            for (int i = 0; i < PER_LANE; ++i) so[warp][j][lane + 32 * i] = o[part * (ROWS / 2) + j][i];
        __syncthreads();
        for (int e = threadIdx.x; e < ROWS / 2 * 32 * PER_LANE; e += ATT_WARPS * 32) {
            const int j = e / (32 * PER_LANE), d = e % (32 * PER_LANE), row = part * (ROWS / 2) + j;
            if (row >= count || d >= head_dim) continue;
            float mm = -INFINITY;
#pragma unroll
            for (int w = 0; w < ATT_WARPS; ++w) mm = fmaxf(mm, sm[w][row]);
            float ltot = 0.0f, acc = 0.0f;
#pragma unroll
            for (int w = 0; w < ATT_WARPS; ++w) {
                const float wt = sl[w][row] > 0.0f ? expf(sm[w][row] - mm) : 0.0f;
                ltot += sl[w][row] * wt;
                acc = fmaf(so[w][j][d], wt, acc);
            }
            const float inv = 1.0f / ltot;
            out[((size_t)(t0 + row) * num_heads + h) * head_dim + d] = from_f32<TQ>(acc * inv);
        }
    }
    if (bad && lane == 0) atomicCAS(status, 0, TI_ERR_BAD_PAGE);
}

}  // namespace

#define TI_DISPATCH_QC(qd, cd, CALL)                                               \
    if (qd == TI_F32 && cd == TI_F32) { CALL(float, float); }                      \
    else if (qd == TI_BF16 && cd == TI_BF16) { CALL(bf16, bf16); }                 \
    else if (qd == TI_F32 && cd == TI_BF16) { CALL(float, bf16); }                 \
    else return ti_fail("attention: dtype codes q=%d cache=%d are not supported", qd, cd);

extern "C" int ti_qk_norm_rope_store(const float* qkv, int qkv_stride, const float* q_weight,
                                     const float* k_weight, float eps, const float* inv_freq,
                                     const int* positions, const int* req_of_tok,
                                     const int* block_table, int bt_stride, void* pages,
                                     int cache_dtype, int num_pages, int page_size, int write_kv,
                                     int num_tokens, int num_heads, int num_kv_heads, int head_dim,
                                     int rotary_dim, void* q_out, int q_dtype, int* status,
                                     void* stream) {
    if (num_tokens == 0) return 0;
    TI_REQUIRE(head_dim >= 1 && head_dim <= MAX_HEAD_DIM,
               "qk_norm_rope_store: head_dim %d must be at most %d", head_dim, MAX_HEAD_DIM);
    TI_REQUIRE(rotary_dim >= 0 && rotary_dim <= head_dim && rotary_dim % 2 == 0,
               "qk_norm_rope_store: the rotated width %d must be even and at most head_dim %d",
               rotary_dim, head_dim);
    TI_REQUIRE(rotary_dim == 0 || inv_freq != nullptr, "qk_norm_rope_store: no rotation table");
    const int items = num_heads + 2 * num_kv_heads;
    dim3 grid(num_tokens, (items + WARPS - 1) / WARPS);
    cudaStream_t s = (cudaStream_t)stream;
    const int half = head_dim / 2;
    int ipw = num_tokens >= 512 ? (items + WARPS - 1) / WARPS : 1;            // vectors per warp
    if (ipw > 8) ipw = 8;
    dim3 vgrid(num_tokens, (items + WARPS * ipw - 1) / (WARPS * ipw));
    // the register kernel pairs element k with k + head_dim / 2: for a rotation over the whole head only
    const int vec = rotary_dim != head_dim ? 0
                    : (half % 4 == 0 && half > 64) ? 4 : (half % 2 == 0 && half <= 64) ? 2 : 0;
#define CALL(TQ, TC)                                                                          \
    if (vec == 2 && ipw == 1)                                                                 \
        ti_launch_pdl((qk_norm_rope_store_one_kernel<TQ, TC, 2>), vgrid, WARPS * 32, 0, s,     \
            qkv, qkv_stride, q_weight, k_weight, eps, inv_freq, positions, req_of_tok, block_table, \
            bt_stride, (TC*)pages, num_pages, page_size, write_kv, num_heads, num_kv_heads,     \
            head_dim, (TQ*)q_out, status);                                                     \
    else if (vec == 4 && ipw == 1)                                                            \
        ti_launch_pdl((qk_norm_rope_store_one_kernel<TQ, TC, 4>), vgrid, WARPS * 32, 0, s,     \
            qkv, qkv_stride, q_weight, k_weight, eps, inv_freq, positions, req_of_tok, block_table, \
            bt_stride, (TC*)pages, num_pages, page_size, write_kv, num_heads, num_kv_heads,     \
            head_dim, (TQ*)q_out, status);                                                     \
    else if (vec == 2)                                                                        \
        ti_launch_pdl(qk_norm_rope_store_vec_kernel<TQ, TC, 2>, vgrid, WARPS * 32, 0, s,       \
            qkv, qkv_stride, q_weight, k_weight, eps, inv_freq, positions, req_of_tok, block_table, \
            bt_stride, (TC*)pages, num_pages, page_size, write_kv, num_heads, num_kv_heads,     \
            head_dim, ipw, (TQ*)q_out, status);                                                \
    else if (vec == 4)                                                                        \
        ti_launch_pdl(qk_norm_rope_store_vec_kernel<TQ, TC, 4>, vgrid, WARPS * 32, 0, s,       \
            qkv, qkv_stride, q_weight, k_weight, eps, inv_freq, positions, req_of_tok, block_table, \
            bt_stride, (TC*)pages, num_pages, page_size, write_kv, num_heads, num_kv_heads,     \
            head_dim, ipw, (TQ*)q_out, status);                                                \
    else                                                                                      \
        ti_launch_pdl(qk_norm_rope_store_kernel<TQ, TC>, grid, WARPS * 32, 0, s,               \
            qkv, qkv_stride, q_weight, k_weight, eps, inv_freq, positions, req_of_tok, block_table, \
            bt_stride, (TC*)pages, num_pages, page_size, write_kv, num_heads, num_kv_heads,     \
            head_dim, rotary_dim, (TQ*)q_out, status)
    TI_DISPATCH_QC(q_dtype, cache_dtype, CALL)
#undef CALL
    return ti_check_launch("qk_norm_rope_store");
}

// `rows` (may be null) lists the tokens to compute; without it all `num_rows` tokens are computed.
extern "C" int ti_paged_attention_simple(const void* q, int q_dtype, const int* rows,
                                         const int* positions,
                                         const int* req_of_tok, const int* block_table,
                                         int bt_stride, const void* pages, int cache_dtype,
                                         int num_pages, int page_size, int num_rows,
                                         int num_heads, int num_kv_heads, int head_dim, int window,
                                         float scale, void* out, int* status, void* stream) {
    if (num_rows == 0) return 0;
    TI_REQUIRE(head_dim >= 1 && head_dim <= MAX_HEAD_DIM,
               "paged_attention: head_dim %d must be at most %d", head_dim, MAX_HEAD_DIM);
    TI_REQUIRE(num_heads % num_kv_heads == 0, "paged_attention: %d heads over %d kv heads",
               num_heads, num_kv_heads);
    dim3 grid(num_rows, num_heads);
    cudaStream_t s = (cudaStream_t)stream;
    // Few blocks wait for their loads, many cover one another's.  us at 8 / 4 / 1 keys ahead, 16 heads of 128: 3 requests
    // with one token at 200 keys (48 blocks) 8.2 / 8.7 / 13, 16 tokens of one at up to 30 keys (256) 4.1 / 4.4 / 4.6, of 8
    // requests 64 tokens each (8,192) 92 / 67 / 59, of 64 requests 16 tokens each (16,384) 111 / 77 / 54 (one key at a time
    // by four warps: 54, 11, 82 and 57)
    int device = 0, sms = 0;
    cudaGetDevice(&device);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    const long long blocks = (long long)num_rows * num_heads;
    const int per_lane = head_dim <= 32 ? 1 : head_dim <= 64 ? 2 : head_dim <= 128 ? 4 : 8;
#define LAUNCH(TQ, TC, N, A)                                                                    \
    ti_launch_pdl(paged_attention_simple_kernel<TQ, TC, N, A>, grid, dim3(ATT_WARPS * 32), 0, s, \
        (const TQ*)q, rows, positions, req_of_tok, block_table, bt_stride, (const TC*)pages,     \
        num_pages, page_size, num_heads, num_kv_heads, head_dim, window, scale, (TQ*)out, status)
#define PICK(TQ, TC, N)                                                                         \
    {                                                                                           \
        if (blocks <= sms) LAUNCH(TQ, TC, N, 8);                                                 \
        else if (blocks <= 2 * sms) LAUNCH(TQ, TC, N, 4);                                        \
        else LAUNCH(TQ, TC, N, 1);                                                               \
    }
#define CALL(TQ, TC)                                                                            \
    if (per_lane == 1) PICK(TQ, TC, 1)                                                           \
    else if (per_lane == 2) PICK(TQ, TC, 2)                                                      \
    else if (per_lane == 4) PICK(TQ, TC, 4)                                                      \
    else PICK(TQ, TC, 8)
    TI_DISPATCH_QC(q_dtype, cache_dtype, CALL)
#undef CALL
#undef PICK
#undef LAUNCH
    return ti_check_launch("paged_attention_simple");
}

// The tokens of `tiles` (int32 [num_tiles, 3] = {request row, first flat token, at most tile_rows tokens}, consecutive tokens of
// one request), without a window: the bits of ti_paged_attention_simple.
extern "C" int ti_paged_attention_portions(const void* q, int q_dtype, const int* tiles, int num_tiles, int tile_rows,
                                           const int* positions, const int* block_table, int bt_stride, const void* pages,
                                           int cache_dtype, int num_pages, int page_size, int num_heads, int num_kv_heads,
                                           int head_dim, float scale, void* out, int* status, void* stream) {
    if (num_tiles == 0) return 0;
    TI_REQUIRE(head_dim >= 1 && head_dim <= MAX_HEAD_DIM, "paged_attention: head_dim %d must be at most %d", head_dim,
               MAX_HEAD_DIM);
    TI_REQUIRE(num_heads % num_kv_heads == 0, "paged_attention: %d heads over %d kv heads", num_heads, num_kv_heads);
    TI_REQUIRE(tile_rows >= 1, "paged_attention: tiles of %d rows", tile_rows);
    const int runs = (tile_rows + ROWS - 1) / ROWS;
    const dim3 grid((unsigned)num_heads * num_tiles * runs);
    cudaStream_t s = (cudaStream_t)stream;
    const int per_lane = head_dim <= 32 ? 1 : head_dim <= 64 ? 2 : head_dim <= 128 ? 4 : 8;
#define LAUNCH(TQ, TC, N)                                                                       \
    ti_launch_pdl(paged_attention_rows_kernel<TQ, TC, N>, grid, dim3(ATT_WARPS * 32), 0, s, (const TQ*)q, tiles, runs, positions, \
        block_table, bt_stride, (const TC*)pages, num_pages, page_size, num_heads, num_kv_heads, head_dim, scale, (TQ*)out, \
        status)
#define CALL(TQ, TC)                                                                            \
    if (per_lane == 1) LAUNCH(TQ, TC, 1);                                                        \
    else if (per_lane == 2) LAUNCH(TQ, TC, 2);                                                   \
    else if (per_lane == 4) LAUNCH(TQ, TC, 4);                                                   \
    else LAUNCH(TQ, TC, 8)
    TI_DISPATCH_QC(q_dtype, cache_dtype, CALL)
#undef CALL
#undef LAUNCH
    return ti_check_launch("paged_attention_portions");
}

TI_TAPED(ti_qk_norm_rope_store)
TI_TAPED(ti_paged_attention_simple)
TI_TAPED(ti_paged_attention_portions)

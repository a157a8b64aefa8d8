// Paged attention with optional parts, on the CUDA cores, and the kernels that prepare its heads.
//
//  * qk_rownorm_rope_store: from a float32 product with the columns [queries | keys | values |
//    anything else], norms the whole query row and the whole key row (RMS over all heads at once,
//    one weight per column), turns the first `rot` elements of every head by the token's position
//    (neighbouring elements 2i, 2i + 1 form a pair; angle = position * inv_freq[i]), writes keys
//    and values into the token's page and the queries out.
//  * latent_prepare: from a float32 product with the columns [query heads of (dk plain | dr
//    rotated) | latent of `rank` | one rotated key part of dr]: the latent is normed (RMS, a weight
//    per element) and stored with the turned key part as ONE row of the token's page; the plain
//    query parts and the turned query parts go out separately.
//  * qkv_turn_store: the same columns with the norms of whole rows or none: the first `rot` elements of every query and key
//    head are turned by the token's position (pairs of neighbours, or element i with i + rot/2), the
//    first `v_rot` elements of every value head by frequencies of their own, values may be mixed with another layer's values of the token before
//    that, keys and values go into the token's page and the queries out.  turn_rows turns the heads of finished rows by plus or minus
//    their position (the way back for outputs over turned values) and multiplies by sigmoid(gate).
//  * slice_rmsnorm: the RMS norm (a weight per element) of the first n columns of rows with a stride.
//  * head_project: out[t, h, :] = in[t, h, :] W[h] with a matrix [n_in, n_out] per head.
//  * attention_options: one block per (token, query head).  Token i sees key j <= i when j is not
//    behind the window (i - j < window) and not in an earlier chunk (j >= floor(i / chunk) *
//    chunk); score = (q . k) * scale, times head_scale[h] if given, then cap * tanh(score / cap)
//    if cap > 0; softmax over the visible keys, whose denominator also counts exp(sink[h]) if a
//    sink is given; the normalised output is multiplied by sigmoid(gate), one gate per head or
//    one per output element.  With `shared_rows` a page holds one row of dk elements per token
//    and kv head, and the value of a key is the first dv elements of that row.
//
// All arithmetic is float32 (positions, angles, norms, scores, softmax weights, the weighted sum);
// inputs and outputs may be float32 or bfloat16.  The order in which a row's keys are added
// depends on the row alone, so a row's bits do not depend on the batch or on how a prompt was cut.
// Page layout without `shared_rows`: keys [kv head][slot][dk], behind them values [kv head][slot][dv].
#include "common.cuh"
#include "head_units.cuh"

namespace {

constexpr int WARPS = 4;
enum { TI_ERR_BAD_PAGE = 1 };

// The turn of a head by a table of the token's cosines and sines (`cs[pair]`, made once per token: the angle
// depends on the position and the pair alone, not on the head).  A head of n elements whose first `rot` are
// turned has rot/2 pairs and n - rot single elements: item i < rot/2 is pair i, the others are singles.
struct TurnItem { int a, b; };      // the pair's two elements (b < 0: a single element a)
__device__ __forceinline__ TurnItem turn_item(int i, int rot, int halves) {
    const int half = rot >> 1;
    if (i >= half) return {rot + (i - half), -1};
    return halves ? TurnItem{i, i + half} : TurnItem{2 * i, 2 * i + 1};
}

__device__ __forceinline__ void fill_turn_table(float2* cs, int pairs, float pos, const float* __restrict__ inv_freq,
                                                float mag) {
    for (int i = threadIdx.x; i < pairs; i += blockDim.x) {
        float s, c;
        sincosf(pos * inv_freq[i], &s, &c);
        cs[i] = make_float2(c * mag, s * mag);
    }
}

// What qkv_turn_store does before it turns: an RMS norm over the whole query row and the whole key row with a
// weight per element (or none), and values mixed with another layer's values of the same token.
struct RowNorm { int on; float eps; const float* q_weight; const float* k_weight; };
struct ValueMix { const float* first; int stride; float share; };

__device__ __forceinline__ float row_unit(const float* row, int n, float eps, float* scratch) {
    float ss = 0.0f;
    for (int e = threadIdx.x; e < n; e += blockDim.x) ss = fmaf(row[e], row[e], ss);
    return 1.0f / sqrtf(block_sum(ss, scratch) / (float)n + eps);
}
__device__ __forceinline__ float normed(const float* row, int e, float inv, const float* weight) {
    return weight ? row[e] * inv * weight[e] : row[e] * inv;
}
__device__ __forceinline__ float mixed(const float* row, const float* first, int e, float share) {
    return first ? (1.0f - share) * row[e] + share * first[e] : row[e];
}

template <typename TQ, typename TC>
__global__ void __launch_bounds__(256)
qkv_turn_store_kernel(const float* proj, int stride, const RowNorm norm, const ValueMix mix,
                      const float* inv_freq, int rot, int halves, float mag,
                      const float* v_inv_freq, int v_rot, int v_halves,
                      const int* positions, const int* req_of_tok,
                      const int* block_table, int bt_stride, TC* __restrict__ pages, int num_pages,
                      int page_size, int write_kv, int num_heads, int num_kv_heads, int dk, int dv,
                      TQ* __restrict__ q_out, int* __restrict__ status) {
    pdl_launch();
    pdl_wait();
    __shared__ float scratch[32];
    extern __shared__ float2 turn_table[];             // rot/2 entries for queries and keys, then v_rot/2 for values
    const int t = blockIdx.x;
    const int nq = num_heads * dk, nk = num_kv_heads * dk;
    const float* row = proj + (size_t)t * stride;
    const int pos_i = positions[t];
    const float pos = (float)pos_i;
    float2* cs = turn_table;
    float2* vcs = turn_table + (rot >> 1);
    fill_turn_table(cs, rot >> 1, pos, inv_freq, mag);
    if (write_kv) fill_turn_table(vcs, v_rot >> 1, pos, v_inv_freq, 1.0f);
    const float* krow = row + nq;
    const float inv_q = norm.on ? row_unit(row, nq, norm.eps, scratch) : 1.0f;
    const float inv_k = norm.on && write_kv ? row_unit(krow, nk, norm.eps, scratch) : 1.0f;
    __syncthreads();
    const int per_head = (rot >> 1) + (dk - rot);      // items of a query or key head
    for (int e = threadIdx.x; e < num_heads * per_head; e += blockDim.x) {
        const int h = e / per_head, i = e % per_head;
        const TurnItem it = turn_item(i, rot, halves);
        const int at = h * dk;
        TQ* dst = q_out + (size_t)t * nq + at;
        const float a = normed(row, at + it.a, inv_q, norm.q_weight);
        if (it.b < 0) { dst[it.a] = from_f32<TQ>(a); continue; }
        const float b = normed(row, at + it.b, inv_q, norm.q_weight);
        const float2 f = cs[i];
        dst[it.a] = from_f32<TQ>(a * f.x - b * f.y);
        dst[it.b] = from_f32<TQ>(b * f.x + a * f.y);
    }
    if (!write_kv) return;
    const int page = block_table[(size_t)req_of_tok[t] * bt_stride + pos_i / page_size];
    if (page < 0 || page >= num_pages) {
        if (threadIdx.x == 0) atomicCAS(status, 0, TI_ERR_BAD_PAGE);
        return;
    }
    const int slot = pos_i % page_size;
    TC* base = pages + (size_t)page * num_kv_heads * page_size * (dk + dv);
    for (int e = threadIdx.x; e < num_kv_heads * per_head; e += blockDim.x) {
        const int g = e / per_head, i = e % per_head;
        const TurnItem it = turn_item(i, rot, halves);
        const int at = g * dk;
        TC* dst = base + ((size_t)g * page_size + slot) * dk;
        const float a = normed(krow, at + it.a, inv_k, norm.k_weight);
        if (it.b < 0) { dst[it.a] = from_f32<TC>(a); continue; }
        const float b = normed(krow, at + it.b, inv_k, norm.k_weight);
        const float2 f = cs[i];
        dst[it.a] = from_f32<TC>(a * f.x - b * f.y);
        dst[it.b] = from_f32<TC>(b * f.x + a * f.y);
    }
    TC* vbase = base + (size_t)num_kv_heads * page_size * dk;
    const float* vrow = krow + nk;
    const float* first = mix.first ? mix.first + (size_t)t * mix.stride : nullptr;
    const int v_per_head = (v_rot >> 1) + (dv - v_rot);
    for (int e = threadIdx.x; e < num_kv_heads * v_per_head; e += blockDim.x) {
        const int g = e / v_per_head, i = e % v_per_head;
        const TurnItem it = turn_item(i, v_rot, v_halves);
        const int at = g * dv;
        TC* dst = vbase + ((size_t)g * page_size + slot) * dv;
        const float a = mixed(vrow, first, at + it.a, mix.share);
        if (it.b < 0) { dst[it.a] = from_f32<TC>(a); continue; }
        const float b = mixed(vrow, first, at + it.b, mix.share);
        const float2 f = vcs[i];
        dst[it.a] = from_f32<TC>(a * f.x - b * f.y);
        dst[it.b] = from_f32<TC>(b * f.x + a * f.y);
    }
}

// The same where heads and turned widths fall into units of four elements: a thread keeps NU units of the query
// and key row in registers, so that the row is read once, four elements a load; cosines, sines and the page are looked
// up before the wait, values go through while the norms' loads are on their way, and both norms' sums meet at one
// barrier.  One block per token; what bounds it is the block's chain of latencies, once in a step of single tokens and as
// often as blocks follow one another on an SM for many.  AHEAD: the weights are asked for before the wait; many tokens
// rather have more blocks an SM.  16 query and 4 key heads, norms over whole rows, us element by element (a sine per
// element) -> now at one and 2,048 tokens: heads of 64 5.6 -> 2.9, 19.4 -> 14.2, of 128 8.6 -> 3.3, 33 -> 17.8 (with
// blocks of 512 threads 26.1).
struct RowHeads {
    const float* proj; int stride;
    RowNorm norm; ValueMix mix;
    const float* inv_freq; int rot, halves; float mag;
    const float* v_inv_freq; int v_rot, v_halves;
    const int* positions; const int* req_of_tok; const int* block_table; int bt_stride;
    int num_pages, page_size, write_kv, num_heads, num_kv_heads, dk, dv;
};

template <typename TQ, typename TC, int THREADS, int NU, bool AHEAD>
__global__ void __launch_bounds__(THREADS, 1024 / THREADS)
row_heads_units_kernel(const RowHeads p, TC* __restrict__ pages, TQ* __restrict__ q_out, int* __restrict__ status) {
    extern __shared__ __align__(16) float2 turn_table[];
    constexpr int SHARES = NU / 2, SUMS = SHARES * THREADS / 32;
    __shared__ float sums[2][SUMS];
    const int t = blockIdx.x, tid = threadIdx.x, pos = p.positions[t];
    const int hu = p.dk >> 2, qu = p.num_heads * hu, total = qu + (p.write_kv ? p.num_kv_heads * hu : 0);
    const int nq = p.num_heads * p.dk, nk = p.num_kv_heads * p.dk;
    float2* vcs = turn_table + (p.rot >> 1);
    pdl_launch();
    fill_turn_table(turn_table, p.rot >> 1, (float)pos, p.inv_freq, p.mag);
    TC* page = nullptr;                                // the token's page: keys of head 0
    if (p.write_kv) {
        fill_turn_table(vcs, p.v_rot >> 1, (float)pos, p.v_inv_freq, 1.0f);
        const int id = p.block_table[(size_t)p.req_of_tok[t] * p.bt_stride + pos / p.page_size];
        if (id >= 0 && id < p.num_pages) page = pages + (size_t)id * p.num_kv_heads * p.page_size * (p.dk + p.dv);
        else if (tid == 0) atomicCAS(status, 0, TI_ERR_BAD_PAGE);
    }
    const int slot = pos % p.page_size;
    // unit i: its head (query heads, behind them key heads) and its place there
    auto head_of = [&](int i) { return i / hu; };
    auto place_of = [&](int i) { return i - i / hu * hu; };
    auto weight_of = [&](int i) {
        const float* weight = i < qu ? p.norm.q_weight : p.norm.k_weight;
        if (i >= total || !p.norm.on || !weight) return make_float4(1.0f, 1.0f, 1.0f, 1.0f);
        const int u = place_of(i);
        return load_unit(weight + (head_of(i) - (i < qu ? 0 : p.num_heads)) * p.dk, u, u < p.rot >> 2, p.halves, p.rot >> 1);
    };
    float4 w[NU], x[NU];
    if (AHEAD) {
#pragma unroll
        for (int j = 0; j < NU; ++j) w[j] = weight_of(tid + THREADS * j);
    }
    __syncthreads();                                   // the turn tables
    pdl_wait();
    const float* row = p.proj + (size_t)t * p.stride;
#pragma unroll
    for (int j = 0; j < NU; ++j) {
        const int i = tid + THREADS * j;
        x[j] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (i < total) {
            const int u = place_of(i);
            x[j] = load_unit(row + head_of(i) * p.dk, u, u < p.rot >> 2, p.halves, p.rot >> 1);
        }
    }
    if (page) {
        const int vu = p.dv >> 2;
        const float* first = p.mix.first ? p.mix.first + (size_t)t * p.mix.stride : nullptr;
        TC* values = page + (size_t)p.num_kv_heads * p.page_size * p.dk;
        for (int i = tid; i < p.num_kv_heads * vu; i += THREADS) {
            const int g = i / vu, u = i - g * vu;
            const bool turned = u < p.v_rot >> 2;
            float4 v = load_unit(row + nq + nk + g * p.dv, u, turned, p.v_halves, p.v_rot >> 1);
            if (first) {
                const float4 f = load_unit(first + g * p.dv, u, turned, p.v_halves, p.v_rot >> 1);
                const float own = 1.0f - p.mix.share;
                v = make_float4(own * v.x + p.mix.share * f.x, own * v.y + p.mix.share * f.y, own * v.z + p.mix.share * f.z,
                                own * v.w + p.mix.share * f.w);
            }
            if (turned) v = turn_unit(v, vcs, u);
            store_unit<TC>(values + ((size_t)g * p.page_size + slot) * p.dv, u, turned, p.v_halves, p.v_rot >> 1, v);
        }
    }
    float inv_q = 1.0f, inv_k = 1.0f;
    if (p.norm.on) {
        // Four units a thread are summed as the two threads of twice as wide a block sum them: a row's bits must not depend
        // on the number of tokens, which chooses between the two.
#pragma unroll
        for (int p0 = 0; p0 < SHARES; ++p0) {
            float2 ss = make_float2(0.0f, 0.0f);       // of the query row, of the key row
#pragma unroll
            for (int j = p0; j < NU; j += SHARES) {
                const float s = fmaf(x[j].w, x[j].w, fmaf(x[j].z, x[j].z, fmaf(x[j].y, x[j].y, x[j].x * x[j].x)));
                if (tid + THREADS * j < qu) ss.x += s; else ss.y += s;
            }
            ss = make_float2(warp_sum(ss.x), warp_sum(ss.y));
            const int at = p0 * (THREADS / 32) + (tid >> 5);
            if ((tid & 31) == 0) { sums[0][at] = ss.x; sums[1][at] = ss.y; }
        }
        __syncthreads();
        float2 ss = make_float2(0.0f, 0.0f);
#pragma unroll
        for (int i = 0; i < SUMS; ++i) { ss.x += sums[0][i]; ss.y += sums[1][i]; }
        inv_q = 1.0f / sqrtf(ss.x / (float)nq + p.norm.eps);
        inv_k = 1.0f / sqrtf(ss.y / (float)nk + p.norm.eps);
    }
#pragma unroll
    for (int j = 0; j < NU; ++j) {
        const int i = tid + THREADS * j;
        if (i >= total) break;
        const int h = head_of(i), u = place_of(i);
        const bool turned = u < p.rot >> 2;
        const float inv = i < qu ? inv_q : inv_k;
        float4 v = x[j];
        if (p.norm.on) {
            if (!AHEAD) w[j] = weight_of(i);
            v = make_float4(v.x * inv * w[j].x, v.y * inv * w[j].y, v.z * inv * w[j].z, v.w * inv * w[j].w);
        }
        if (turned) v = turn_unit(v, turn_table, u);
        if (i < qu) store_unit<TQ>(q_out + (size_t)t * nq + h * p.dk, u, turned, p.halves, p.rot >> 1, v);
        else if (page) store_unit<TC>(page + ((size_t)(h - p.num_heads) * p.page_size + slot) * p.dk, u, turned, p.halves,
                                      p.rot >> 1, v);
    }
}

// x[t, h, :] turned by sign * position over its first `rot` elements, then times sigmoid(gate[t, h * n + j]); a
// block per token, a thread reads and writes both elements of a pair, so the rows may be turned in place
template <typename T>
__global__ void __launch_bounds__(256)
turn_rows_kernel(const T* x, const int* positions, const float* inv_freq, int rot,
                 int halves, float sign, const float* gate, int gate_stride, int num_heads, int n, T* out) {
    pdl_launch();
    pdl_wait();
    extern __shared__ float2 turn_table[];
    const int t = blockIdx.x;
    fill_turn_table(turn_table, rot >> 1, sign * (float)positions[t], inv_freq, 1.0f);
    __syncthreads();
    const int per_head = (rot >> 1) + (n - rot);
    const float* gt = gate ? gate + (size_t)t * gate_stride : nullptr;
    for (int e = threadIdx.x; e < num_heads * per_head; e += blockDim.x) {
        const int h = e / per_head, i = e % per_head;
        const TurnItem it = turn_item(i, rot, halves);
        const size_t at = ((size_t)t * num_heads + h) * n;
        const float a = to_f32(x[at + it.a]);
        if (it.b < 0) {
            out[at + it.a] = from_f32<T>(gt ? a / (1.0f + expf(-gt[(size_t)h * n + it.a])) : a);
            continue;
        }
        const float b = to_f32(x[at + it.b]);
        const float2 f = turn_table[i];
        float ya = a * f.x - b * f.y, yb = b * f.x + a * f.y;
        if (gt) {
            ya *= 1.0f / (1.0f + expf(-gt[(size_t)h * n + it.a]));
            yb *= 1.0f / (1.0f + expf(-gt[(size_t)h * n + it.b]));
        }
        out[at + it.a] = from_f32<T>(ya);
        out[at + it.b] = from_f32<T>(yb);
    }
}

// out[t, :] = x[t, :n] / sqrt(mean(x[t, :n]^2) + eps) * w over rows with a stride: the norm of a column slice of a
// product (a latent that shares its product with other columns)
template <typename TO>
__global__ void __launch_bounds__(256)
slice_rmsnorm_kernel(const float* x, int stride, int n, const float* w, float eps, TO* __restrict__ out) {
    pdl_launch();
    pdl_wait();
    __shared__ float scratch[32];
    const float* row = x + (size_t)blockIdx.x * stride;
    float ss = 0.0f;
    for (int e = threadIdx.x; e < n; e += blockDim.x) ss = fmaf(row[e], row[e], ss);
    const float inv = 1.0f / sqrtf(block_sum(ss, scratch) / (float)n + eps);
    for (int e = threadIdx.x; e < n; e += blockDim.x)
        out[(size_t)blockIdx.x * n + e] = from_f32<TO>(row[e] * inv * (w ? w[e] : 1.0f));
}

// Grid: tokens x 2; the first block of a token has its query heads, the second its latent and key part.  UNITS: all parts
// are multiples of four elements on aligned rows, which then travel four at a time, a thread's loads together.  Cosines
// and sines are made before the wait, once per token instead of once per head.  16 heads, latent of 512: one token 6.6 ->
// 1.9 us, 2,048 tokens 23.4 -> 9.7.
template <typename TQ, typename TC, bool UNITS>
__global__ void __launch_bounds__(256)
latent_prepare_kernel(const float* qproj, int q_stride, const float* proj, int stride,
                      const float* latent_weight, float eps,
                      const float* inv_freq, float mag, const int* positions,
                      const int* req_of_tok, const int* block_table, int bt_stride,
                      TC* __restrict__ pages, int num_pages, int page_size, int num_heads, int dk, int dr,
                      int rank, TQ* __restrict__ q_plain, TQ* __restrict__ q_full, int* __restrict__ status) {
    extern __shared__ __align__(16) float2 cs[];
    __shared__ float scratch[32];
    const int t = blockIdx.x, tid = threadIdx.x, pos = positions[t];
    const int qh = dk + dr, row_len = rank + dr;
    pdl_launch();
    fill_turn_table(cs, dr >> 1, (float)pos, inv_freq, mag);
    __syncthreads();
    auto pair = [&](const float* x, int j) {             // element j of the turned part x
        const float2 f = cs[j >> 1];
        return (j & 1) ? x[j] * f.x + x[j ^ 1] * f.y : x[j] * f.x - x[j ^ 1] * f.y;
    };
    if (blockIdx.y == 0) {
        pdl_wait();
        const float* row = qproj + (size_t)t * q_stride;
        TQ* plain = q_plain + (size_t)t * num_heads * dk;
        TQ* full = q_full + (size_t)t * num_heads * row_len + rank;
        if (UNITS) {
            const int hu = qh >> 2, total = num_heads * hu;
            for (int i0 = tid; i0 < total; i0 += 4 * 256) {
                float4 v[4];
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (i0 + 256 * j < total) v[j] = *reinterpret_cast<const float4*>(row + 4 * (i0 + 256 * j));
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int i = i0 + 256 * j;
                    if (i >= total) break;
                    const int h = i / hu, u = i - h * hu, r = u - (dk >> 2);
                    if (r < 0) {
                        store_unit<TQ>(plain + (size_t)h * dk, u, false, 0, 0, v[j]);
                    } else {
                        const float4 pairs = make_float4(v[j].x, v[j].z, v[j].y, v[j].w);
                        store_unit<TQ>(full + (size_t)h * row_len, r, true, 0, 0, turn_unit(pairs, cs, r));
                    }
                }
            }
        } else {
            for (int e = tid; e < num_heads * qh; e += 256) {
                const int j = e % qh, h = e / qh;
                if (j < dk) plain[(size_t)h * dk + j] = from_f32<TQ>(row[e]);
                else full[(size_t)h * row_len + (j - dk)] = from_f32<TQ>(pair(row + h * qh + dk, j - dk));
            }
        }
        return;
    }
    const int page = block_table[(size_t)req_of_tok[t] * bt_stride + pos / page_size];
    pdl_wait();
    if (page < 0 || page >= num_pages) {
        if (tid == 0) atomicCAS(status, 0, TI_ERR_BAD_PAGE);
        return;
    }
    TC* dst = pages + ((size_t)page * page_size + pos % page_size) * row_len;
    const float* lat = proj + (size_t)t * stride;
    if (UNITS && rank <= 4 * 256) {                      // the latent in registers: read once
        const bool mine = 4 * tid < rank;
        float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (mine) v = *reinterpret_cast<const float4*>(lat + 4 * tid);
        for (int r = tid; r < dr >> 2; r += 256)
            store_unit<TC>(dst + rank, r, true, 0, 0, turn_unit(load_unit(lat + rank, r, true, 0, 0), cs, r));
        const float ss = fmaf(v.w, v.w, fmaf(v.z, v.z, fmaf(v.y, v.y, v.x * v.x)));
        const float inv = 1.0f / sqrtf(block_sum(ss, scratch) / (float)rank + eps);
        if (!mine) return;
        float4 w = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
        if (latent_weight) w = *reinterpret_cast<const float4*>(latent_weight + 4 * tid);
        store_unit<TC>(dst, tid, false, 0, 0, make_float4(v.x * inv * w.x, v.y * inv * w.y, v.z * inv * w.z, v.w * inv * w.w));
        return;
    }
    float ss = 0.0f;
    for (int e = tid; e < rank; e += 256) ss = fmaf(lat[e], lat[e], ss);
    const float inv = 1.0f / sqrtf(block_sum(ss, scratch) / (float)rank + eps);
    for (int e = tid; e < rank; e += 256)
        dst[e] = from_f32<TC>(lat[e] * inv * (latent_weight ? latent_weight[e] : 1.0f));
    for (int e = tid; e < dr; e += 256) dst[rank + e] = from_f32<TC>(pair(lat + rank, e));
}

// out[t, h, n] = sum_k in[t, h, k] * w[h, k, n], bfloat16, for few tokens: a block has up to TT tokens of one head and 32
// columns, a thread four neighbouring columns (8 bytes of a weight row a load) and every 32nd k.  What bounds it is the
// weights' way from memory, so all blocks of a head together ask for all of them at once, and up to KP rows a thread
// before the wait for the kernel before; the tokens' inputs lie in shared memory with the tokens of one k side by side,
// and the threads' sums meet by shuffles and in shared memory in a fixed order.  16 heads, us at one token: 128 -> 512
// 5.7 -> 2.7, 512 -> 128 15.5 -> 2.9 (blocks of 128 columns: 16 of them, an eighth of k a warp).
constexpr int HP_TOKENS = 16;      // most tokens of a block
constexpr int HP_COLS = 32, HP_GROUPS = 32, HP_THREADS = HP_COLS / 4 * HP_GROUPS;

__device__ __forceinline__ uint2 load4(const bf16* p, bool whole, int left) {
    if (whole) return *reinterpret_cast<const uint2*>(p);
    bf16 v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = i < left ? p[i] : __float2bfloat16_rn(0.0f);
    const __nv_bfloat162 lo = __halves2bfloat162(v[0], v[1]), hi = __halves2bfloat162(v[2], v[3]);
    return make_uint2(*reinterpret_cast<const unsigned*>(&lo), *reinterpret_cast<const unsigned*>(&hi));
}

template <int TT, int KP>
__global__ void __launch_bounds__(HP_THREADS)
head_project_few_kernel(const bf16* in, int in_stride_t, int in_stride_h, const bf16* __restrict__ w, int n_in,
                        int n_out, bf16* out, int out_stride_t, int out_stride_h, int num_tokens, int vec_ok) {
    extern __shared__ __align__(16) float xs[];      // [n_in][TT]; afterwards the warps' partial sums [8][TT][HP_COLS]
    const int t0 = blockIdx.x * TT, h = blockIdx.y, tid = threadIdx.x, kg = tid >> 3;
    const int n0 = blockIdx.z * HP_COLS + (tid & 7) * 4;
    const int nt = min(TT, num_tokens - t0), left = n_out - n0;
    const bool whole = vec_ok && left >= 4;
    const bf16* wh = w + (size_t)h * n_in * n_out + n0;
    pdl_launch();
    uint2 wv[KP];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int i = 0; i < KP; ++i) {
            const int k = k0 + kg + HP_GROUPS * i;
            wv[i] = make_uint2(0u, 0u);
            if (k < n_in && left > 0) wv[i] = load4(wh + (size_t)k * n_out, whole, left);
        }
    };
    fetch(0);
    pdl_wait();
    for (int k = tid; k < n_in; k += HP_THREADS) {
        const bf16* src = in + (size_t)t0 * in_stride_t + (size_t)h * in_stride_h + k;
        float x[TT];                                 // all tokens' loads together
#pragma unroll
        for (int tt = 0; tt < TT; ++tt) x[tt] = tt < nt ? to_f32(src[(size_t)tt * in_stride_t]) : 0.0f;
#pragma unroll
        for (int tt = 0; tt < TT; tt += 4) store4(xs + k * TT + tt, make_float4(x[tt], x[tt + 1], x[tt + 2], x[tt + 3]));
    }
    __syncthreads();
    float acc[TT][4];
#pragma unroll
    for (int i = 0; i < TT; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.0f;
    for (int k0 = 0; k0 < n_in; k0 += HP_GROUPS * KP) {
        if (k0) fetch(k0);
#pragma unroll
        for (int i = 0; i < KP; ++i) {
            const int k = k0 + kg + HP_GROUPS * i;
            if (k >= n_in) break;
            const __nv_bfloat162 lo = *reinterpret_cast<const __nv_bfloat162*>(&wv[i].x);
            const __nv_bfloat162 hi = *reinterpret_cast<const __nv_bfloat162*>(&wv[i].y);
            const float wf[4] = {__bfloat162float(lo.x), __bfloat162float(lo.y), __bfloat162float(hi.x), __bfloat162float(hi.y)};
            const float4* x4 = reinterpret_cast<const float4*>(xs + k * TT);
#pragma unroll
            for (int q = 0; q < TT / 4; ++q) {
                const float4 x = x4[q];
                const float xv[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
                for (int a = 0; a < 4; ++a)
#pragma unroll
                    for (int c = 0; c < 4; ++c) acc[4 * q + a][c] = fmaf(xv[a], wf[c], acc[4 * q + a][c]);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < TT; ++i)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            acc[i][c] += __shfl_xor_sync(0xffffffffu, acc[i][c], 8);
            acc[i][c] += __shfl_xor_sync(0xffffffffu, acc[i][c], 16);
        }
    __syncthreads();                                 // the inputs have been read
    if ((tid & 31) < 8) {
#pragma unroll
        for (int i = 0; i < TT; ++i)
            *reinterpret_cast<float4*>(xs + ((tid >> 5) * TT + i) * HP_COLS + (tid & 7) * 4) =
                make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    }
    __syncthreads();
    for (int e = tid; e < nt * HP_COLS; e += HP_THREADS) {
        const int tt = e / HP_COLS, c = e % HP_COLS, n = blockIdx.z * HP_COLS + c;
        if (n >= n_out) continue;
        float sum = 0.0f;
#pragma unroll
        for (int i = 0; i < HP_THREADS / 32; ++i) sum += xs[(i * TT + tt) * HP_COLS + c];
        out[(size_t)(t0 + tt) * out_stride_t + (size_t)h * out_stride_h + n] = __float2bfloat16_rn(sum);
    }
}

// The same product for many tokens, where the grid has blocks enough: four warps, a thread per column,
// all of k in one thread (no meeting of partial sums).
template <typename TI, typename TW, typename TO>
__global__ void __launch_bounds__(128)
head_project_rows_kernel(const TI* in, int in_stride_t, int in_stride_h, const TW* w, int n_in,
                         int n_out, TO* out, int out_stride_t, int out_stride_h, int num_tokens) {
    pdl_launch();
    pdl_wait();
    extern __shared__ __align__(16) float xs[];      // [n_in][HP_TOKENS]
    const int t0 = blockIdx.x * HP_TOKENS, h = blockIdx.y;
    const int n = blockIdx.z * 128 + threadIdx.x;
    const int nt = min(HP_TOKENS, num_tokens - t0);
    for (int e = threadIdx.x; e < HP_TOKENS * n_in; e += 128) {
        const int tt = e / n_in, k = e % n_in;
        xs[k * HP_TOKENS + tt] =
            tt < nt ? to_f32(in[(size_t)(t0 + tt) * in_stride_t + (size_t)h * in_stride_h + k]) : 0.0f;
    }
    __syncthreads();
    if (n >= n_out) return;
    float acc[HP_TOKENS];
#pragma unroll
    for (int i = 0; i < HP_TOKENS; ++i) acc[i] = 0.0f;
    const TW* wh = w + (size_t)h * n_in * n_out + n;
#pragma unroll 4
    for (int k = 0; k < n_in; ++k) {
        const float wv = to_f32(wh[(size_t)k * n_out]);
        const float4* x4 = reinterpret_cast<const float4*>(xs + k * HP_TOKENS);
#pragma unroll
        for (int i = 0; i < HP_TOKENS / 4; ++i) {
            const float4 x = x4[i];
            acc[4 * i] = fmaf(x.x, wv, acc[4 * i]);
            acc[4 * i + 1] = fmaf(x.y, wv, acc[4 * i + 1]);
            acc[4 * i + 2] = fmaf(x.z, wv, acc[4 * i + 2]);
            acc[4 * i + 3] = fmaf(x.w, wv, acc[4 * i + 3]);
        }
    }
#pragma unroll
    for (int i = 0; i < HP_TOKENS; ++i)
        if (i < nt) out[(size_t)(t0 + i) * out_stride_t + (size_t)h * out_stride_h + n] = from_f32<TO>(acc[i]);
}

struct AttnOptions {
    int window, chunk;            // 0: none
    float scale, softcap;         // softcap 0: none
    const float* head_scale;      // [heads] or null
    const float* sink;            // [heads] or null
    const float* gate;            // [T, gate_stride] float32 or null
    int gate_stride, gate_per_head, shared_rows;
};

template <typename TQ, typename TC, int PER_LANE>
__global__ void __launch_bounds__(WARPS * 32)
attention_options_kernel(const TQ* q, const int* __restrict__ rows, const int* __restrict__ positions,
                         const int* __restrict__ req_of_tok, const int* __restrict__ block_table,
                         int bt_stride, const TC* pages, int num_pages, int page_size, int num_heads,
                         int num_kv_heads, int dk, int dv, AttnOptions opt, TQ* __restrict__ out,
                         int* __restrict__ status) {
    __shared__ float so[WARPS][PER_LANE * 32];
    __shared__ float sm[WARPS], sl[WARPS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int h = blockIdx.y, t = rows ? rows[blockIdx.x] : blockIdx.x;
    const int kvh = h / (num_heads / num_kv_heads);
    const int pos = positions[t];
    const int* table = block_table + (size_t)req_of_tok[t] * bt_stride;
    int lo = opt.window > 0 ? max(0, pos - opt.window + 1) : 0;
    if (opt.chunk > 0) lo = max(lo, pos / opt.chunk * opt.chunk);
    const size_t page_elems = (size_t)num_kv_heads * page_size * (opt.shared_rows ? dk : dk + dv);
    const size_t v_base = opt.shared_rows ? 0 : (size_t)num_kv_heads * page_size * dk;
    const int v_row = opt.shared_rows ? dk : dv;
    const float hs = opt.head_scale ? opt.scale * opt.head_scale[h] : opt.scale;

    float qv[PER_LANE], o[PER_LANE];
    const TQ* qh = q + ((size_t)t * num_heads + h) * dk;
#pragma unroll
    for (int i = 0; i < PER_LANE; ++i) {
        const int d = lane + 32 * i;
        qv[i] = d < dk ? to_f32(qh[d]) : 0.0f;
        o[i] = 0.0f;
    }
    // the sink is one more logit without a value; the first warp starts from it
    float m = -INFINITY, l = 0.0f;
    if (opt.sink && warp == 0) { m = opt.sink[h]; l = 1.0f; }
    bool bad = false;
    for (int p = lo + warp; p <= pos; p += WARPS) {
        const int page = table[p / page_size];
        if (page < 0 || page >= num_pages) { bad = true; continue; }
        const TC* base = pages + (size_t)page * page_elems;
        const TC* kp = base + ((size_t)kvh * page_size + p % page_size) * dk;
        const TC* vp = base + v_base + ((size_t)kvh * page_size + p % page_size) * v_row;
        float s = 0.0f;
#pragma unroll
        for (int i = 0; i < PER_LANE; ++i) {
            const int d = lane + 32 * i;
            if (d < dk) s = fmaf(qv[i], to_f32(kp[d]), s);
        }
        s = warp_sum(s) * hs;
        if (opt.softcap > 0.0f) s = opt.softcap * tanhf(s / opt.softcap);
        const float m_new = fmaxf(m, s);
        const float alpha = expf(m - m_new);
        const float pr = expf(s - m_new);
        l = l * alpha + pr;
#pragma unroll
        for (int i = 0; i < PER_LANE; ++i) {
            const int d = lane + 32 * i;
            if (d < dv) o[i] = fmaf(pr, to_f32(vp[d]), o[i] * alpha);
        }
        m = m_new;
    }
    if (bad && lane == 0) atomicCAS(status, 0, TI_ERR_BAD_PAGE);
#pragma unroll
    for (int i = 0; i < PER_LANE; ++i) so[warp][lane + 32 * i] = o[i];
    if (lane == 0) { sm[warp] = m; sl[warp] = l; }
    __syncthreads();
    if (warp == 0) {
        float mm = -INFINITY;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) mm = fmaxf(mm, sm[w]);
        float ltot = 0.0f, wt[WARPS];
#pragma unroll
        for (int w = 0; w < WARPS; ++w) {
            wt[w] = sl[w] > 0.0f ? expf(sm[w] - mm) : 0.0f;
            ltot += sl[w] * wt[w];
        }
        const float inv = 1.0f / ltot;
        TQ* oh = out + ((size_t)t * num_heads + h) * dv;
        const float* gt = opt.gate ? opt.gate + (size_t)t * opt.gate_stride : nullptr;
        const float head_gate = (gt && opt.gate_per_head) ? 1.0f / (1.0f + expf(-gt[h])) : 1.0f;
        for (int d = lane; d < dv; d += 32) {
            float acc = 0.0f;
#pragma unroll
            for (int w = 0; w < WARPS; ++w) acc = fmaf(so[w][d], wt[w], acc);
            acc *= inv * head_gate;
            if (gt && !opt.gate_per_head) acc *= 1.0f / (1.0f + expf(-gt[(size_t)h * dv + d]));
            oh[d] = from_f32<TQ>(acc);
        }
    }
}

}  // namespace

#define TI_DISPATCH_QC(qd, cd, CALL)                                               \
    if (qd == TI_F32 && cd == TI_F32) { CALL(float, float); }                      \
    else if (qd == TI_BF16 && cd == TI_BF16) { CALL(bf16, bf16); }                 \
    else if (qd == TI_F32 && cd == TI_BF16) { CALL(float, bf16); }                 \
    else return ti_fail("attention: dtype codes q=%d cache=%d are not supported", qd, cd);

// Rows of whole heads (RowHeads) to pages and queries: in units of four elements where the sizes and addresses allow it
// and the query and key rows together fit into two units a thread of a block, else element by element.
static int launch_row_heads(const char* what, const RowHeads& p, int num_tokens, void* pages, int cache_dtype, void* q_out,
                            int q_dtype, int* status, cudaStream_t s) {
    auto aligned = [](const void* x) { return (uintptr_t)x % 16 == 0; };
    const size_t smem = (size_t)(p.rot / 2 + p.v_rot / 2) * sizeof(float2);      // the token's cosines and sines
    TI_REQUIRE(smem <= 47 * 1024, "%s: rotated widths %d and %d", what, p.rot, p.v_rot);
    const int units = (p.num_heads + p.num_kv_heads) * p.dk / 4;
    const bool fits = p.dk % 4 == 0 && p.dv % 4 == 0 && p.rot % 4 == 0 && p.v_rot % 4 == 0 && p.stride % 4 == 0 &&
                      (p.mix.first == nullptr || p.mix.stride % 4 == 0) && units <= 2048 && aligned(p.proj) &&
                      aligned(p.norm.q_weight) && aligned(p.norm.k_weight) && aligned(p.mix.first) && aligned(pages) &&
                      aligned(q_out);
#define UNITS(TQ, TC, N, NU, AHEAD)                                                                                             \
    ti_launch_pdl((row_heads_units_kernel<TQ, TC, N, NU, AHEAD>), dim3(num_tokens), dim3(N), smem, s, p, (TC*)pages, (TQ*)q_out, status)
#define CALL(TQ, TC)                                                                                                 \
    if (!fits)                                                                                                       \
        ti_launch_pdl((qkv_turn_store_kernel<TQ, TC>), dim3(num_tokens), dim3(256), smem, s, p.proj, p.stride, p.norm, \
                      p.mix, p.inv_freq, p.rot, p.halves, p.mag, p.v_inv_freq, p.v_rot, p.v_halves, p.positions,       \
                      p.req_of_tok, p.block_table, p.bt_stride, (TC*)pages, p.num_pages, p.page_size, p.write_kv,      \
                      p.num_heads, p.num_kv_heads, p.dk, p.dv, (TQ*)q_out, status);                                    \
    else if (units <= 512) UNITS(TQ, TC, 256, 2, true);                                                              \
    else if (units <= 1024 && num_tokens < 256) UNITS(TQ, TC, 512, 2, true);                                         \
    else if (units <= 1024) UNITS(TQ, TC, 256, 4, false);                                                            \
    else UNITS(TQ, TC, 1024, 2, true)
    TI_DISPATCH_QC(q_dtype, cache_dtype, CALL)
#undef CALL
#undef UNITS
    return ti_check_launch(what);
}

extern "C" int ti_heads_prepare_store(const float* proj, int stride, const float* bias, const float* q_weight,
                                      const float* k_weight, int pre_norm, int post_norm, float eps,
                                      const float* inv_freq, int rot, int halves, float mag, float temp_coef,
                                      int temp_every, int values_from_keys, const int* positions,
                                      const int* req_of_tok, const int* block_table, int bt_stride, void* pages,
                                      int cache_dtype, int num_pages, int page_size, int write_kv, int num_tokens,
                                      int num_heads, int num_kv_heads, int dk, int dv, void* q_out, int q_dtype,
                                      int* status, void* stream);

extern "C" int ti_qk_rownorm_rope_store(const float* proj, int stride, const float* q_weight,
                                        const float* k_weight, float eps, const float* inv_freq, int rot,
                                        const int* positions, const int* req_of_tok, const int* block_table,
                                        int bt_stride, void* pages, int cache_dtype, int num_pages,
                                        int page_size, int write_kv, int num_tokens, int num_heads,
                                        int num_kv_heads, int dk, int dv, int per_head, void* q_out, int q_dtype,
                                        int* status, void* stream) {
    if (num_tokens == 0) return 0;
    TI_REQUIRE(rot >= 0 && rot <= dk && rot % 2 == 0, "qk_rownorm_rope_store: rotated width %d must be even "
               "and at most the head size %d", rot, dk);
    TI_REQUIRE(rot == 0 || inv_freq != nullptr, "qk_rownorm_rope_store: a rotation needs its frequencies");
    TI_REQUIRE(q_dtype == cache_dtype || q_dtype == TI_F32, "qk_rownorm_rope_store: dtype codes q=%d cache=%d are not "
               "supported", q_dtype, cache_dtype);
    if (per_head)                                       // heads normed one by one: head_rows.cu
        return ti_heads_prepare_store(proj, stride, nullptr, q_weight, k_weight, 1, 0, eps, inv_freq, rot, 0, 1.0f, 0.0f, 0, 0,
                                      positions, req_of_tok, block_table, bt_stride, pages, cache_dtype, num_pages, page_size,
                                      write_kv, num_tokens, num_heads, num_kv_heads, dk, dv, q_out, q_dtype, status, stream);
    const RowHeads p{proj, stride, {1, eps, q_weight, k_weight}, {nullptr, 0, 0.0f}, inv_freq, rot, 0, 1.0f, nullptr, 0, 0,
                     positions, req_of_tok, block_table, bt_stride, num_pages, page_size, write_kv, num_heads, num_kv_heads,
                     dk, dv};
    return launch_row_heads("qk_rownorm_rope_store", p, num_tokens, pages, cache_dtype, q_out, q_dtype, status,
                            (cudaStream_t)stream);
}

extern "C" int ti_slice_rmsnorm(const float* x, int stride, int num_rows, int n, const float* weight, float eps,
                                void* out, int out_dtype, void* stream) {
    if (num_rows == 0 || n == 0) return 0;
    cudaStream_t s = (cudaStream_t)stream;
    if (out_dtype == TI_BF16) ti_launch_pdl(slice_rmsnorm_kernel<bf16>, dim3(num_rows), dim3(256), 0, s, x, stride, n,
                                            weight, eps, (bf16*)out);
    else if (out_dtype == TI_F32) ti_launch_pdl(slice_rmsnorm_kernel<float>, dim3(num_rows), dim3(256), 0, s, x,
                                                stride, n, weight, eps, (float*)out);
    else return ti_fail("slice_rmsnorm: output dtype code %d", out_dtype);
    return ti_check_launch("slice_rmsnorm");
}

// `qproj` holds a token's query heads of (dk plain | dr rotated), `proj` its latent of `rank` and the key part of dr
extern "C" int ti_latent_prepare(const float* qproj, int q_stride, const float* proj, int stride,
                                 const float* latent_weight, float eps,
                                 const float* inv_freq, float mag, const int* positions, const int* req_of_tok,
                                 const int* block_table, int bt_stride, void* pages, int cache_dtype,
                                 int num_pages, int page_size, int num_tokens, int num_heads, int dk, int dr,
                                 int rank, void* q_plain, void* q_full, int q_dtype, int* status,
                                 void* stream) {
    if (num_tokens == 0) return 0;
    TI_REQUIRE(dr >= 0 && dr % 2 == 0, "latent_prepare: the rotated width %d must be even", dr);
    TI_REQUIRE(dr == 0 || inv_freq != nullptr, "latent_prepare: a rotation needs its frequencies");
    cudaStream_t s = (cudaStream_t)stream;
    auto aligned = [](const void* x) { return (uintptr_t)x % 16 == 0; };
    const size_t smem = (size_t)(dr / 2) * sizeof(float2);
    TI_REQUIRE(smem <= 47 * 1024, "latent_prepare: a rotated width of %d", dr);
    const bool units = dk % 4 == 0 && dr % 4 == 0 && rank % 4 == 0 && q_stride % 4 == 0 && stride % 4 == 0 && aligned(qproj) &&
                       aligned(proj) && aligned(latent_weight) && aligned(pages) && aligned(q_plain) && aligned(q_full);
#define CALL(TQ, TC)                                                                              \
    ti_launch_pdl((units ? latent_prepare_kernel<TQ, TC, true> : latent_prepare_kernel<TQ, TC, false>), dim3(num_tokens, 2), \
        dim3(256), smem, s, qproj, q_stride, proj, stride, latent_weight, eps, inv_freq, mag, positions, req_of_tok,  \
        block_table, bt_stride, (TC*)pages, num_pages, page_size, num_heads, dk, dr, rank, (TQ*)q_plain, (TQ*)q_full, status)
    TI_DISPATCH_QC(q_dtype, cache_dtype, CALL)
#undef CALL
    return ti_check_launch("latent_prepare");
}

extern "C" int ti_qkv_turn_store(const float* proj, int stride, int row_norm, float eps, const float* q_weight,
                                 const float* k_weight, const float* mix_first, int mix_stride, float mix_share,
                                 const float* inv_freq, int rot, int halves, float mag,
                                 const float* v_inv_freq, int v_rot, int v_halves, const int* positions,
                                 const int* req_of_tok, const int* block_table, int bt_stride, void* pages,
                                 int cache_dtype, int num_pages, int page_size, int write_kv, int num_tokens,
                                 int num_heads, int num_kv_heads, int dk, int dv, void* q_out, int q_dtype,
                                 int* status, void* stream) {
    if (num_tokens == 0) return 0;
    TI_REQUIRE(rot >= 0 && rot <= dk && rot % 2 == 0, "qkv_turn_store: rotated width %d must be even and at most "
               "the head size %d", rot, dk);
    TI_REQUIRE(v_rot >= 0 && v_rot <= dv && v_rot % 2 == 0, "qkv_turn_store: rotated width %d of the values must be "
               "even and at most their head size %d", v_rot, dv);
    TI_REQUIRE((rot == 0 || inv_freq != nullptr) && (v_rot == 0 || v_inv_freq != nullptr),
               "qkv_turn_store: a rotation needs its frequencies");
    const RowHeads p{proj, stride, {row_norm, eps, q_weight, k_weight}, {mix_first, mix_stride, mix_share}, inv_freq, rot,
                     halves, mag, v_inv_freq, v_rot, v_halves, positions, req_of_tok, block_table, bt_stride, num_pages,
                     page_size, write_kv, num_heads, num_kv_heads, dk, dv};
    return launch_row_heads("qkv_turn_store", p, num_tokens, pages, cache_dtype, q_out, q_dtype, status, (cudaStream_t)stream);
}

extern "C" int ti_turn_rows(const void* x, int dtype, const int* positions, const float* inv_freq, int rot, int halves,
                            float sign, const float* gate, int gate_stride, int num_tokens, int num_heads, int n,
                            void* out, void* stream) {
    if (num_tokens == 0 || num_heads == 0) return 0;
    TI_REQUIRE(rot >= 0 && rot <= n && rot % 2 == 0, "turn_rows: rotated width %d must be even and at most %d", rot, n);
    TI_REQUIRE(rot == 0 || inv_freq != nullptr, "turn_rows: a rotation needs its frequencies");
    const size_t smem = (size_t)(rot / 2) * sizeof(float2);
    TI_REQUIRE(smem <= 48 * 1024, "turn_rows: a rotated width of %d", rot);
    cudaStream_t s = (cudaStream_t)stream;
    if (dtype == TI_BF16)
        ti_launch_pdl(turn_rows_kernel<bf16>, dim3(num_tokens), dim3(256), smem, s, (const bf16*)x, positions,
                      inv_freq, rot, halves, sign, gate, gate_stride, num_heads, n, (bf16*)out);
    else if (dtype == TI_F32)
        ti_launch_pdl(turn_rows_kernel<float>, dim3(num_tokens), dim3(256), smem, s, (const float*)x, positions,
                      inv_freq, rot, halves, sign, gate, gate_stride, num_heads, n, (float*)out);
    else return ti_fail("turn_rows: dtype code %d", dtype);
    return ti_check_launch("turn_rows");
}

extern "C" int ti_head_project(const void* in, int in_dtype, int in_stride_t, int in_stride_h, const void* w,
                               int w_dtype, int n_in, int n_out, void* out, int out_dtype, int out_stride_t,
                               int out_stride_h, int num_tokens, int num_heads, void* stream) {
    if (num_tokens == 0 || num_heads == 0) return 0;
    TI_REQUIRE(in_dtype == out_dtype, "head_project: input and output must have one dtype");
    const size_t smem = (size_t)HP_TOKENS * n_in * sizeof(float);
    TI_REQUIRE(smem <= 48 * 1024, "head_project: %d inputs per head are more than the kernel stages", n_in);
    cudaStream_t s = (cudaStream_t)stream;
    // Up to 64 tokens in bfloat16 (a step of single tokens): the form whose threads split k, so that a head's weights are
    // on their way at once; else a thread per column with all of k.  (A row's bits can differ between the two forms;
    // within a form they depend on the row alone.)  Float32 rows always take the second form: their bits must not depend
    // on the step around them.
    if (in_dtype == TI_BF16 && w_dtype == TI_BF16 && num_tokens <= 64) {
        const int vec_ok = n_out % 4 == 0 && (uintptr_t)w % 8 == 0;      // four columns a load
        const int tt = num_tokens <= 4 ? 4 : num_tokens <= 8 ? 8 : 16;
        const dim3 grid((num_tokens + tt - 1) / tt, num_heads, (n_out + HP_COLS - 1) / HP_COLS);
        const size_t inputs = (size_t)tt * n_in * sizeof(float), meet = (size_t)(HP_THREADS / 32) * tt * HP_COLS * sizeof(float);
#define LAUNCH(TT, KP)                                                                                              \
    ti_launch_pdl((head_project_few_kernel<TT, KP>), grid, dim3(HP_THREADS), inputs > meet ? inputs : meet, s,        \
        (const bf16*)in, in_stride_t, in_stride_h, (const bf16*)w, n_in, n_out, (bf16*)out, out_stride_t, out_stride_h, \
        num_tokens, vec_ok)
        if (n_in <= HP_GROUPS * 4) {
            if (tt == 4) LAUNCH(4, 4); else if (tt == 8) LAUNCH(8, 4); else LAUNCH(16, 4);
        } else {
            if (tt == 4) LAUNCH(4, 16); else if (tt == 8) LAUNCH(8, 16); else LAUNCH(16, 16);
        }
#undef LAUNCH
        return ti_check_launch("head_project");
    }
    dim3 grid((num_tokens + HP_TOKENS - 1) / HP_TOKENS, num_heads, (n_out + 127) / 128);
#define CALL(TI_, TW_)                                                                            \
    ti_launch_pdl((head_project_rows_kernel<TI_, TW_, TI_>), dim3(grid), dim3(128), smem, s,        \
        (const TI_*)in, in_stride_t, in_stride_h, (const TW_*)w, n_in, n_out, (TI_*)out,            \
        out_stride_t, out_stride_h, num_tokens)
    if (in_dtype == TI_F32 && w_dtype == TI_F32) { CALL(float, float); }
    else if (in_dtype == TI_F32 && w_dtype == TI_BF16) { CALL(float, bf16); }
    else if (in_dtype == TI_BF16 && w_dtype == TI_BF16) { CALL(bf16, bf16); }
    else return ti_fail("head_project: dtype codes in=%d w=%d are not supported", in_dtype, w_dtype);
#undef CALL
    return ti_check_launch("head_project");
}

// `rows` (may be null) lists the tokens to compute; without it all `num_rows` tokens are computed.
extern "C" int ti_attention_options(const void* q, int q_dtype, const int* rows, const int* positions,
                                    const int* req_of_tok, const int* block_table, int bt_stride,
                                    const void* pages, int cache_dtype, int num_pages, int page_size,
                                    int num_rows, int num_heads, int num_kv_heads, int dk, int dv,
                                    int shared_rows, int window, int chunk, float scale, float softcap,
                                    const float* head_scale, const float* sink, const float* gate,
                                    int gate_stride, int gate_per_head, void* out, int* status,
                                    void* stream) {
    if (num_rows == 0) return 0;
    const int widest = dk > dv ? dk : dv;
    TI_REQUIRE(dk >= 1 && dv >= 1 && widest <= 1024, "attention_options: head sizes %d and %d must be at "
               "most 1024", dk, dv);
    TI_REQUIRE(num_heads % num_kv_heads == 0, "attention_options: %d heads over %d kv heads", num_heads,
               num_kv_heads);
    TI_REQUIRE(!shared_rows || dv <= dk, "attention_options: a value of %d elements does not fit into a "
               "shared row of %d", dv, dk);
    TI_REQUIRE(window >= 0 && chunk >= 0 && softcap >= 0.0f, "attention_options: negative window, chunk or cap");
    AttnOptions opt = {window, chunk, scale, softcap, head_scale, sink, gate, gate_stride, gate_per_head,
                       shared_rows};
    dim3 grid(num_rows, num_heads);
    cudaStream_t s = (cudaStream_t)stream;
#define LAUNCH(TQ, TC, PL)                                                                         \
    attention_options_kernel<TQ, TC, PL><<<grid, WARPS * 32, 0, s>>>(                               \
        (const TQ*)q, rows, positions, req_of_tok, block_table, bt_stride, (const TC*)pages,          \
        num_pages, page_size, num_heads, num_kv_heads, dk, dv, opt, (TQ*)out, status)
#define CALL(TQ, TC)                                                                               \
    if (widest <= 128) LAUNCH(TQ, TC, 4); else if (widest <= 256) LAUNCH(TQ, TC, 8);                 \
    else if (widest <= 640) LAUNCH(TQ, TC, 20); else LAUNCH(TQ, TC, 32)
    TI_DISPATCH_QC(q_dtype, cache_dtype, CALL)
#undef CALL
#undef LAUNCH
    return ti_check_launch("attention_options");
}

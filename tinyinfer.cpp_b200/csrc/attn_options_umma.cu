// Paged flash attention with optional parts for prompt portions on the 5th-generation tensor cores: the same options,
// cache layouts and precision as attn_options_tc.cu (a window and/or chunks, a score factor per head, a cap, a sink, an
// output gate, one shared row per token as key and value), whose mma.sync kernel keeps single tokens and every size
// that this one does not take.
//
// Arrangement.  A block has 128 rows, the MMA's M side: the heads of one kv group of 128 / group consecutive tokens of
// one request, fetched by one 3-D TMA box per 64 elements of the head.  It walks its keys in tiles of 64.  A tile
// comes as chunks of 64 keys x 64 elements (TMA, 128-byte swizzle).  Score products take every key
// chunk as K-major B operand; the value products take the chunks of the block's value columns as MN-major B operand:
// chunks of their own, or with shared rows the very chunks that the scores have used.  Values of more than 256
// columns are cut into slices, a block each.
//
// Softmax weights stay float32 through the second product: a weight is cut into three bfloat16 parts (8 + 8 + 8 bits
// of its significand) which the softmax threads (one per row) write into tensor memory as the A operand of three
// products.  So a tile of 64 keys is K / 16 score products of N = 64 and twelve value products.
//
// What bounds it (clock stamps in the roles).  Latent rows of 576 with 256 value columns: 7,000 cycles a tile, a chain of
// 12 value products (137 each), the reload of the value chunks, the last 16 of 36 score products (98 each, issue as much
// as operand reads) and the softmax; rows of 288: 4,300.  Heads of 128 with a cap: 6,800 a tile and block, of which the
// softmax takes 4,300, two blocks at a time.  16 heads over 2,048 tokens at positions 0 / 2,048, us, against the mma.sync
// kernel: latent 576 258 / 744 against 1,217 / 3,152 (416 / 1,232 with one issuing thread and a barrier per chunk), latent
// 288 91 / 251 against 387 / 916, heads of 128 over 4 kv heads with a cap 132 / 269 against 317 / 766, of 64 with a cap
// 123 / 249 against 210 / 558.  Steps without a portion stay with that kernel: it cuts a row's keys over blocks.
//
// Two forms.  Rows of up to 128 elements with values of their own (NS = 1): two blocks per SM that fill one another's
// gaps, with 256 columns of tensor memory each: outputs up to 128, scores 64, weights 96, of which the last 32 lie where
// the scores were if the outputs take 128.  There the next scores wait for the products with that part (heads of 128
// without a cap, 256 tokens behind 2,000: 91 -> 96 us); a block is the plain chain of scores, softmax, value products.
// Wide shared rows (NS = 2): one block per SM, two score buffers, and the next tile's
// scores issued beside the value products of this one.  Where shared memory holds two tiles (rows up to 320) they wait
// for nothing; where it holds one (576: queries 147 KB, a tile 74 KB) the part of the row that is no value of this
// block comes first, and the rest follows as the value products release its chunks.
//
// Order: warp 0 issues TMA, warp 1 the products (NS = 2: the scores, warp 6 the value products), warps 2-5 are the
// softmax.  Every wait on an mbarrier is bounded: on a timeout the block records status 2, frees its tensor memory and
// returns.
#include <utility>

#include "attn_options.cuh"
#include "sm100.cuh"

namespace {

using namespace sm100;

constexpr int BM = 128, BN = 64;
template <int NS> constexpr int threads_of() { return NS == 1 ? 192 : 224; }
constexpr int QCHUNK = BM * 128, CHUNK = BN * 128;    // bytes: 64 elements of every row
constexpr int MAX_POS = 9;                            // chunks of a tile
constexpr float LOG2E = 1.4426950408889634f;
constexpr float RESCALE_STEP = 8.0f;                  // in log2 units
enum { TI_ERR_BAD_PAGE = 1, TI_ERR_TIMEOUT = 2 };

struct UmmaOptions {
    int window, chunk;
    float scale, softcap;
    const float* head_scale;
    const float* sink;
    const float* gate;
    int gate_stride, gate_per_head;
};

// How a tile is cut: `chunks` of a key row, `places` chunks of a tile, the last `nv` of them the value chunks of a slice.
struct Shape {
    int dk, dv, chunks, places, nv, slices, stages, shared, run;
};

__device__ __forceinline__ int first_visible(int p, const UmmaOptions& o) { return first_key_seen(p, o.window, o.chunk); }
// D (+)= A B with A from tensor memory (rows in lanes, two bfloat16 of K per 32-bit column).
__device__ __forceinline__ void umma_bf16_tmem_a(unsigned tmem_d, unsigned tmem_a, unsigned long long db, unsigned idesc,
                                                 unsigned accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n"
        ::"r"(tmem_d), "r"(tmem_a), "l"(db), "r"(idesc), "r"(accumulate) : "memory");
}
// 16 consecutive 32-bit columns of this thread's lane; completion is awaited by the caller.
__device__ __forceinline__ void tmem_store16(unsigned taddr, const unsigned (&v)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};\n"
        ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
          "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
        : "memory");
}
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, void* bar, int x, int y, int z) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];\n"
        ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z) : "memory");
}

// tiles[i] = {request row, first flat token, tokens (<= BM / group)}; NV: chunks of value columns (NS = 1)
template <int NS, int NV>
__global__ void __launch_bounds__(threads_of<NS>(), NS == 1 ? 2 : 1)
attn_options_umma_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_kv,
                         const __grid_constant__ CUtensorMap map_8, const __grid_constant__ CUtensorMap map_1,
                         const int* __restrict__ tiles, const int* __restrict__ positions,
                         const int* __restrict__ block_table, int bt_stride, int num_pages, int page_size, int num_heads,
                         int num_kv_heads, Shape sh, UmmaOptions opt, bf16* __restrict__ out, int* __restrict__ status) {
    constexpr unsigned TMEM_COLS = NS == 1 ? 256 : 512;
    // Columns of tensor memory: outputs from 0 on, scores, the three parts of the weights (32 columns each).  128 columns
    // of outputs (NS = 1) leave no room for the last part, which lies where the scores were.
    constexpr bool LO_IN_SCORES = NS == 1 && NV == 2;
    constexpr unsigned S_AT = NS == 2 ? 256 : NV * 64, HI_AT = S_AT + NS * BN, MID_AT = HI_AT + 32;
    constexpr unsigned LO_AT = LO_IN_SCORES ? S_AT : MID_AT + 32;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    unsigned char* ring = smem + sh.chunks * QCHUNK;
    unsigned long long* bars = (unsigned long long*)(ring + sh.stages * sh.places * CHUNK);
    unsigned long long* q_full = bars;
    unsigned long long* s_full = bars + 1;            // [NS]
    unsigned long long* s_empty = bars + 3;           // [NS]
    unsigned long long* p_full = bars + 5;
    unsigned long long* p_empty = bars + 6;           // value products done: weights may be rewritten, O is up to date
    unsigned long long* full = bars + 7;              // [stages][2]: the chunks only the scores read, the value chunks
    unsigned long long* empty = bars + 11;
    unsigned long long* lo_read = bars + 15;          // LO_IN_SCORES: the products with the last part of the weights are done
    unsigned* tmem_slot = (unsigned*)(bars + 16);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int slice = blockIdx.x % sh.slices, kvh = blockIdx.x / sh.slices;
    const int group = num_heads / num_kv_heads;
    const int req = tiles[blockIdx.y * 3], tok0 = tiles[blockIdx.y * 3 + 1], ntok = tiles[blockIdx.y * 3 + 2];
    const int pos_first = positions[tok0], pos_last = pos_first + ntok - 1;
    const int kv_lo = first_visible(pos_first, opt);
    const int kt_lo = kv_lo / BN, num_kt = pos_last / BN + 1 - kt_lo;
    const int early = sh.places - sh.nv;              // places whose chunks only the scores read
    // shared rows: the chunk of the row at place p
    auto chunk_at = [&](int p) { return p >= early ? slice * sh.nv + p - early : p < slice * sh.nv ? p : p + sh.nv; };

    if (threadIdx.x == 0) {
        mbar_init(q_full, 1);
        for (int i = 0; i < 2; ++i) { mbar_init(&s_full[i], 1); mbar_init(&s_empty[i], 4); }
        mbar_init(p_full, 4);
        mbar_init(p_empty, 1);
        mbar_init(lo_read, 1);
        for (int i = 0; i < 2 * sh.stages; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
        mbar_fence_init();
    }
    if (warp == 1) tmem_alloc(tmem_slot, TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem_base = *tmem_slot;
    pdl_wait();        // queries, keys, values and gates come from the kernels before (the next is not released early)

    bool ok = true;
    if (warp == 0) {
        const int* table = block_table + (size_t)req * bt_stride;
        const int per_page = num_kv_heads * page_size * (sh.shared ? 1 : 2);      // rows of a page in the pool's 2-D view
        const int oob_row = num_pages * per_page;                                 // outside the tensor: zeros
        const int to_v = num_kv_heads * page_size;                                // keys -> values of a page
        if (lane == 0) {
            const int tokens = BM / group;
            mbar_expect_tx(q_full, sh.chunks * tokens * group * 128);
            for (int c = 0; c < sh.chunks; ++c)
                tma_load_3d(smem + c * QCHUNK, &map_q, q_full, c * 64, kvh * group, tok0);
        }
        for (int j = 0; j < num_kt && ok; ++j) {
            const int st = j % sh.stages, phase = (j / sh.stages) & 1;
            const int base = (kt_lo + j) * BN, from_row = kv_lo - base, to_row = pos_last + 1 - base;
            // where `height` rows of the tile from row `at` on begin in the pool
            auto place = [&](int at, int height) {
                const int key0 = base + at;
                if (at >= to_row || at + height <= from_row) return oob_row;
                const int pg = table[key0 / page_size];
                if (pg >= 0 && pg < num_pages) return pg * per_page + kvh * page_size + key0 % page_size;
                atomicCAS(status, 0, TI_ERR_BAD_PAGE);
                return oob_row;
            };
            // this lane's rows of the tile: a run of keys
            const CUtensorMap* map = &map_kv;
            bool mine = lane < BN / sh.run;
            int at = lane * sh.run, row = mine ? place(at, sh.run) : oob_row;
            for (int part = early > 0 ? 0 : 1; part < 2; ++part) {
                if (part == 1 && (from_row > 0 || to_row < BN)) {
                    // Values outside the keys that this block's queries see must be zeros: behind the request's last token
                    // a page may hold what an earlier request left, and a weight of zero times an infinity is not zero.
                    // They come in groups of eight rows, a group at either end row by row (lanes 8 to 15, 16 to 23).
                    const int cut = to_row < BN && to_row % 8 ? to_row / 8 : -1;
                    const int cut_lo = from_row > 0 && from_row % 8 && from_row / 8 != cut ? from_row / 8 : -1;
                    const int eight = lane < 8 ? lane : lane < 16 ? cut : cut_lo;
                    map = lane < 8 ? &map_8 : &map_1;
                    mine = lane < 8 ? lane != cut && lane != cut_lo : lane < 24 && eight >= 0;
                    at = eight * 8 + (lane < 8 ? 0 : lane % 8);
                    row = mine ? place(at, lane < 8 ? 8 : 1) : oob_row;
                }
                unsigned long long* bar = &full[st * 2 + part];
                const int from = part == 0 ? 0 : early, to = part == 0 ? early : sh.places;
                if (lane == 0) {
                    ok = mbar_wait(&empty[st * 2 + part], phase ^ 1);
                    if (ok) mbar_expect_tx(bar, (to - from) * CHUNK);
                }
                ok = __shfl_sync(0xffffffffu, ok, 0);
                if (!ok) break;
                if (!mine) continue;
                for (int p = from; p < to; ++p) {
                    int c, y = row;
                    if (sh.shared) {                  // the row's chunks outside the slice, then the slice's
                        c = chunk_at(p);
                    } else {
                        c = p < sh.chunks ? p : slice * sh.nv + p - sh.chunks;
                        if (p >= sh.chunks && row != oob_row) y = row + to_v;
                    }
                    tma_load_2d(ring + (st * sh.places + p) * CHUNK + at * 128, map, bar, c * 64, y);
                }
            }
        }
    } else if (warp == 1 || warp == 6) {
        // Scores and value products, by one thread (NS = 1) or by two (NS = 2: the scores' 36 products of a tile of 576
        // take a thread longer to issue than to run).  Products into different accumulators may run in another order
        // than they are issued in, so the next scores, where they replace the last part of the weights, wait for the
        // products that read it; the products with the other two parts keep the tensor cores busy meanwhile.
        if (lane == 0) {
            const unsigned idesc_s = umma_idesc(BM, BN);
            const unsigned idesc_o = umma_idesc(BM, sh.nv * 64, /*b_mn_major=*/true);
            const unsigned long long dq = umma_desc(smem), dr = umma_desc(ring), dv_ = umma_desc(ring, CHUNK, 1024);
            // scores of tile j from the chunks of one part; a last chunk of fewer than 64 elements is filled up with zeros
            auto scores = [&](int j, int part) {
                const int st = j % sh.stages, phase = (j / sh.stages) & 1;
                const int from = part == 0 ? 0 : early, to = part == 0 ? early : sh.places;
                if (!ok || from == to) return;
                ok = mbar_wait(&full[st * 2 + part], phase);
                if (!ok) return;
                tc_fence_after();
                const unsigned to_s = tmem_base + S_AT + (NS == 1 ? 0 : (j & 1) * BN);
                unsigned long long b = dr + (unsigned long long)((st * sh.places + from) * (CHUNK >> 4));
                for (int p = from; p < to; ++p, b += CHUNK >> 4) {
                    const unsigned long long a = dq + (unsigned long long)((sh.shared ? chunk_at(p) : p) * (QCHUNK >> 4));
                    umma_bf16(to_s, a, b, idesc_s, p > 0);
#pragma unroll
                    for (int kk = 1; kk < 4; ++kk) umma_bf16(to_s, a + kk * 2, b + kk * 2, idesc_s, 1);
                }
                if (part == 0) umma_commit(&empty[st * 2]);
            };
            auto all_scores = [&](int j) {
                scores(j, 0);
                if (sh.shared) scores(j, 1);
                if (ok) umma_commit(&s_full[NS == 1 ? 0 : j & 1]);
            };
            auto value_products = [&](int j) {
                const int st = j % sh.stages;
                if (ok) ok = mbar_wait(p_full, j & 1);
                if (ok) ok = mbar_wait(&full[st * 2 + 1], (j / sh.stages) & 1);
                if (!ok) return;
                tc_fence_after();
                const unsigned long long b = dv_ + (unsigned long long)((st * sh.places + early) * (CHUNK >> 4));
#pragma unroll
                for (int part = 2; part >= 0; --part) {                                   // the smallest parts first
                    const unsigned a = tmem_base + (part == 2 ? LO_AT : part == 1 ? MID_AT : HI_AT);
#pragma unroll
                    for (int ks = 0; ks < BN / 16; ++ks)
                        umma_bf16_tmem_a(tmem_base, a + ks * 8, b + (unsigned long long)(ks * (2048 >> 4)), idesc_o,
                                         j > 0 || part < 2 || ks > 0);
                    if (LO_IN_SCORES && part == 2) umma_commit(lo_read);
                }
                umma_commit(&empty[st * 2 + 1]);
                umma_commit(p_empty);
            };
            if (warp == 1) {
                ok = mbar_wait(q_full, 0);
                if (ok) tc_fence_after();
                for (int j = 0; j < num_kt && ok; ++j) {
                    if (NS == 2) {
                        // value chunks are read by the value products too, which may still run: a part of the scores
                        // waits for nothing but its own copies
                        ok = mbar_wait(&s_empty[j & 1], ((j >> 1) & 1) ^ 1);
                        if (ok) all_scores(j);
                    } else {
                        if (j == 0) all_scores(0);
                        value_products(j);
                        if (ok && j + 1 < num_kt) {
                            if (LO_IN_SCORES) ok = mbar_wait(lo_read, j & 1);
                            if (ok) all_scores(j + 1);
                        }
                    }
                }
            } else {
                for (int j = 0; j < num_kt && ok; ++j) value_products(j);
            }
        }
    } else {
        const int quarter = warp & 3;                                             // tensor-memory lanes
        const int row = quarter * 32 + lane;
        const int tok = row / group, h = kvh * group + row % group;
        const bool live = tok < ntok;
        const int pos_row = live ? pos_first + tok : -1;                          // -1: sees nothing
        const int lo_row = live ? first_visible(pos_row, opt) : 0;
        const int lo_last = first_visible(pos_last, opt);
        const unsigned lane_addr = (unsigned)(quarter * 32) << 16;
        const float cap_l2e = opt.softcap * LOG2E;
        // one factor per score: into the cap's exponent, or into log2 units
        const float scale = opt.scale * (opt.head_scale && live ? opt.head_scale[h] : 1.0f) *
                            (opt.softcap > 0.0f ? 2.0f * LOG2E / opt.softcap : LOG2E);
        float m_ref = -INFINITY, l_run = 0.0f;
        for (int j = 0; j < num_kt && ok; ++j) {
            const int b = NS == 1 ? 0 : j & 1;
            const int key_lo = (kt_lo + j) * BN;
            ok = mbar_wait(&s_full[b], (NS == 1 ? j : j >> 1) & 1);
            if (!ok) break;
            tc_fence_after();
            float v[BN];
#pragma unroll
            for (int c = 0; c < 2; ++c)
                tmem_load32(tmem_base + lane_addr + S_AT + b * BN + c * 32, *reinterpret_cast<float(*)[32]>(&v[c * 32]));
            if (NS == 2) {
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&s_empty[b]);
            }
            if (opt.softcap > 0.0f) {                 // cap tanh(v / cap) = cap (1 - 2 / (exp(2 v / cap) + 1))
#pragma unroll
                for (int i = 0; i < BN; ++i)
                    v[i] = cap_l2e * fmaf(-2.0f, rcp_approx(ex2_approx(v[i] * scale) + 1.0f), 1.0f);
            } else {
#pragma unroll
                for (int i = 0; i < BN; ++i) v[i] *= scale;
            }
            if (key_lo + BN - 1 > pos_first || key_lo < lo_last) {
#pragma unroll
                for (int i = 0; i < BN; ++i)
                    if (key_lo + i > pos_row || key_lo + i < lo_row) v[i] = -INFINITY;
            }
            float m4[4] = {v[0], v[1], v[2], v[3]};
#pragma unroll
            for (int i = 4; i < BN; i += 4)
#pragma unroll
                for (int u = 0; u < 4; ++u) m4[u] = fmaxf(m4[u], v[i + u]);
            const float m_new = fmaxf(m_ref, fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3])));
            const bool grow = m_new > m_ref + RESCALE_STEP;                       // also true when m_ref is still -inf
            if (j > 0) {
                ok = mbar_wait(p_empty, (j - 1) & 1);
                if (!ok) break;
                tc_fence_after();      // behind the value products, which have read the weights that this tile's replace
                if (__any_sync(0xffffffffu, grow)) {
                    // the output so far was built against m_ref: bring it to the new reference
                    const float factor = grow ? exp2f(m_ref - m_new) : 1.0f;      // 0 if m_ref was -inf
                    l_run *= factor;
#pragma unroll 1
                    for (int c = 0; c < sh.nv * 2; ++c) {
                        float o[32];
                        tmem_load32(tmem_base + lane_addr + c * 32, o);
#pragma unroll
                        for (int i = 0; i < 32; ++i) o[i] *= factor;
                        tmem_store32(tmem_base + lane_addr + c * 32, o);
                    }
                }
            }
            if (grow) m_ref = m_new;
            const float m_use = m_ref == -INFINITY ? 0.0f : m_ref;
            float sum[2] = {0.0f, 0.0f};
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                unsigned hi[16], mid[16], lo[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const float p0 = ex2_approx(v[c * 32 + 2 * i] - m_use), p1 = ex2_approx(v[c * 32 + 2 * i + 1] - m_use);
                    sum[0] += p0;
                    sum[1] += p1;
                    split3_pair(p0, p1, hi[i], mid[i], lo[i]);
                }
                tmem_store16(tmem_base + lane_addr + HI_AT + c * 16, hi);
                tmem_store16(tmem_base + lane_addr + MID_AT + c * 16, mid);
                tmem_store16(tmem_base + lane_addr + LO_AT + c * 16, lo);
            }
            l_run += sum[0] + sum[1];
            asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(p_full);
        }
        if (ok) ok = mbar_wait(p_empty, (num_kt - 1) & 1);
        if (ok) {
            tc_fence_after();
            const size_t t = (size_t)tok0 + tok;
            float l = l_run;
            if (opt.sink && live) l += exp2f(opt.sink[h] * LOG2E - m_ref);
            float inv = 1.0f / l;
            const float* gt = opt.gate && live ? opt.gate + t * opt.gate_stride : nullptr;
            if (gt && opt.gate_per_head) inv *= 1.0f / (1.0f + expf(-gt[h]));
            const float* ge = gt && !opt.gate_per_head ? gt + (size_t)h * sh.dv + slice * sh.nv * 64 : nullptr;
            bf16* orow = out + (t * num_heads + h) * sh.dv + slice * sh.nv * 64;
#pragma unroll 1
            for (int c = 0; c < sh.nv * 2; ++c) {
                float v[32];
                tmem_load32(tmem_base + lane_addr + c * 32, v);
                if (!live) continue;
                unsigned packed[16];
#pragma unroll
                for (int i = 0; i < 32; i += 2) {
                    float a = v[i] * inv, d = v[i + 1] * inv;
                    if (ge) {
                        a *= 1.0f / (1.0f + expf(-ge[c * 32 + i]));
                        d *= 1.0f / (1.0f + expf(-ge[c * 32 + i + 1]));
                    }
                    __nv_bfloat162 pk = __floats2bfloat162_rn(a, d);
                    packed[i >> 1] = *reinterpret_cast<unsigned*>(&pk);
                }
#pragma unroll
                for (int q8 = 0; q8 < 2; ++q8)            // whole 32-byte sectors (a row of outputs is 128-byte aligned)
                    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(orow + c * 32 + q8 * 16),
                                 "r"(packed[q8 * 8]), "r"(packed[q8 * 8 + 1]), "r"(packed[q8 * 8 + 2]),
                                 "r"(packed[q8 * 8 + 3]), "r"(packed[q8 * 8 + 4]), "r"(packed[q8 * 8 + 5]),
                                 "r"(packed[q8 * 8 + 6]), "r"(packed[q8 * 8 + 7]) : "memory");
            }
        }
    }
    if (!ok) atomicCAS(status, 0, TI_ERR_TIMEOUT);
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, TMEM_COLS);
    }
}

size_t smem_bytes(const Shape& sh) {
    return 1024 + (size_t)sh.chunks * QCHUNK + (size_t)sh.stages * sh.places * CHUNK + 17 * 8;
}

// The cut of the rows, or `places` = 0 where the kernel does not take them.
Shape shape_of(int dk, int dv, int page_size, int shared, int group) {
    Shape sh = {};
    if (group < 1 || group > BM || dk < 16 || dk % 16 || dv < 64 || dv % 64 || page_size < 16 || page_size % 16) return sh;
    sh.dk = dk;
    sh.dv = dv;
    sh.shared = shared;
    sh.chunks = (dk + 63) / 64;
    if (shared) {
        if (dv > dk || (dv > 256 && dv % 256)) return sh;
        sh.nv = dv > 256 ? 4 : dv / 64;
    } else {
        if (dk != dv || dv > 128) return sh;
        sh.nv = dv / 64;
    }
    sh.slices = dv / (sh.nv * 64);
    sh.run = BN;
    while (page_size % sh.run) sh.run /= 2;
    const int places = shared ? sh.chunks : sh.chunks + sh.nv;
    if (places > MAX_POS) return sh;
    sh.places = places;
    sh.stages = 2;
    if (smem_bytes(sh) > 227 * 1024) sh.stages = 1;
    if (smem_bytes(sh) > 227 * 1024 || (!shared && sh.stages == 1)) sh.places = 0;
    return sh;
}

int make_map(CUtensorMap* map, const void* base, int rank, const cuuint64_t* dims, const cuuint64_t* strides,
             const cuuint32_t* box) {
    EncodeTiled fn = encode_fn();
    if (!fn) return ti_fail("attn_options_umma: the driver lacks cuTensorMapEncodeTiled");
    const cuuint32_t elem[3] = {1, 1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, rank, const_cast<void*>(base), dims, strides, box, elem,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return ti_fail("attn_options_umma: cuTensorMapEncodeTiled failed with %d", (int)r);
    return 0;
}

}  // namespace

// Query tokens of a block, or 0 where the kernel does not take these sizes.
extern "C" int ti_attn_options_umma_tokens(int dk, int dv, int page_size, int shared_rows, int num_heads, int num_kv_heads) {
    if (num_kv_heads < 1 || num_heads % num_kv_heads) return 0;
    return shape_of(dk, dv, page_size, shared_rows, num_heads / num_kv_heads).places ? BM / (num_heads / num_kv_heads) : 0;
}

// q: bfloat16 [num_tokens, num_heads, dk], out: bfloat16 [num_tokens, num_heads, dv], contiguous.  tiles: int32
// [num_tiles, 3] = {request row, first flat token, tokens}, at most ti_attn_options_umma_tokens consecutive tokens of
// one request each.  The rest as in ti_attn_options_tc.
extern "C" int ti_attn_options_umma(const void* q, const int* tiles, int num_tiles, int num_tokens, const int* positions,
                                    const int* block_table, int bt_stride, const void* pages, int num_pages,
                                    int page_size, int num_heads, int num_kv_heads, int dk, int dv, int shared_rows,
                                    int window, int chunk, float scale, float softcap, const float* head_scale,
                                    const float* sink, const float* gate, int gate_stride, int gate_per_head, void* out,
                                    int* status, void* stream) {
    if (num_tiles == 0) return 0;
    TI_REQUIRE(ti_attn_options_umma_tokens(dk, dv, page_size, shared_rows, num_heads, num_kv_heads) > 0,
               "attn_options_umma: head sizes %d and %d, page size %d or %d heads over %d kv heads are not supported", dk,
               dv, page_size, num_heads, num_kv_heads);
    TI_REQUIRE((uintptr_t)q % 16 == 0 && (uintptr_t)pages % 16 == 0 && (uintptr_t)out % 32 == 0,
               "attn_options_umma: queries and pages must be 16-byte aligned, the output 32-byte");
    TI_REQUIRE(num_tiles <= 65535, "attn_options_umma: %d tiles exceed the grid limit", num_tiles);
    const int group = num_heads / num_kv_heads;
    const Shape sh = shape_of(dk, dv, page_size, shared_rows, group);
    const long long pool_rows = (long long)num_pages * num_kv_heads * page_size * (shared_rows ? 1 : 2);
    TI_REQUIRE(pool_rows < (1LL << 31) - 1, "attn_options_umma: the page pool has too many token slots");
    CUtensorMap map_q, map_kv, map_8, map_1;
    const cuuint64_t qdims[3] = {(cuuint64_t)dk, (cuuint64_t)num_heads, (cuuint64_t)num_tokens};
    const cuuint64_t qstrides[2] = {(cuuint64_t)dk * 2, (cuuint64_t)num_heads * dk * 2};
    const cuuint32_t qbox[3] = {64, (cuuint32_t)group, (cuuint32_t)(BM / group)};
    if (int rc = make_map(&map_q, q, 3, qdims, qstrides, qbox)) return rc;
    const cuuint64_t kdims[2] = {(cuuint64_t)dk, (cuuint64_t)pool_rows};
    const cuuint64_t kstrides[1] = {(cuuint64_t)dk * 2};
    for (auto [map, rows] : {std::pair<CUtensorMap*, int>{&map_kv, sh.run}, {&map_8, 8}, {&map_1, 1}}) {
        const cuuint32_t kbox[2] = {64, (cuuint32_t)rows};
        if (int rc = make_map(map, pages, 2, kdims, kstrides, kbox)) return rc;
    }
    UmmaOptions opt = {window, chunk, scale, softcap, head_scale, sink, gate, gate_stride, gate_per_head};
    const size_t smem = smem_bytes(sh);
    const dim3 grid(num_kv_heads * sh.slices, num_tiles);
    cudaStream_t s = (cudaStream_t)stream;
#define LAUNCH(NS, NV)                                                                                            \
    {                                                                                                             \
        static TiPerDevice configured;                                                                            \
        if (configured.first_use()) {                                                                             \
            cudaError_t e = cudaFuncSetAttribute(attn_options_umma_kernel<NS, NV>,                                 \
                                                 cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);         \
            if (e != cudaSuccess) return ti_fail("attn_options_umma: %s", cudaGetErrorString(e));                  \
            configured.mark();                                                                                    \
        }                                                                                                         \
        ti_launch_pdl(attn_options_umma_kernel<NS, NV>, grid, dim3(threads_of<NS>()), smem, s, map_q, map_kv,      \
                      map_8, map_1, tiles, positions, block_table, bt_stride, num_pages, page_size, num_heads, num_kv_heads, sh, \
                      opt, (bf16*)out, status);                                                                   \
    }
    if (shared_rows) LAUNCH(2, 0) else if (sh.nv == 1) LAUNCH(1, 1) else LAUNCH(1, 2)
#undef LAUNCH
    return ti_check_launch("attn_options_umma");
}
